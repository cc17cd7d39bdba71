// Row-wise steps of a layer stack whose residual stream is one fp32 row per token.
//
//  resid_step    : closes a sublayer and opens the next one.  result (of routed experts: the sum of the rows that the routes
//                  name) -> sigmoid gate -> norm -> added to the stream;
//                  optionally the stream becomes a weighted sum of the kept streams of all layers so far (depth average);
//                  then the norm that feeds the next sublayer.  With `tokens` the stream starts from the embedding.
//  polynorm      : activation a N(z) + b N(z^2) + c N(z^3) + e, N = division by the row's root mean square
//  gate_mul      : result x sigmoid(gate)
//  head_norm_gate: per-head RMS norm x weight x sigmoid(gate)
//  side_act      : gelu_tanh(projection) x a layer's part of the token's second embedding
//  softcap_rows  : cap tanh(x / cap) in place
//  gather_rows   : picks rows of an activation matrix by index
#include <cooperative_groups.h>

#include "ds41_stack.cuh"
#include "ds41_tma.h"

namespace ds41 {

namespace cg = cooperative_groups;

// (mean, sum of squared deviations, count) of a set of values
struct Moments {
  float mean, m2, n;
};
__device__ __forceinline__ Moments merge(Moments a, Moments b) {
  if (b.n == 0.f) return a;
  const float n = a.n + b.n;
  // halves of equal size in all but a row's last pieces: no division in the chain of merges that every row waits for twice
  // (1 row of 2048 columns, layer norms: 11.1 us with the divisions, 10.0 without; 8 rows, RMS norms: 6.6 and 5.8)
  const float d = b.mean - a.mean, f = b.n == a.n ? 0.5f : b.n / n;
  return {fmaf(d, f, a.mean), fmaf(d * d, a.n * f, a.m2 + b.m2), n};
}
__device__ __forceinline__ Moments merge_lanes(Moments v) {          // result in lane 0, then in every lane
#pragma unroll
  for (int o = 16; o; o >>= 1)
    v = merge(v, {__shfl_down_sync(0xffffffffu, v.mean, o), __shfl_down_sync(0xffffffffu, v.m2, o),
                  __shfl_down_sync(0xffffffffu, v.n, o)});
  return {__shfl_sync(0xffffffffu, v.mean, 0), __shfl_sync(0xffffffffu, v.m2, 0), __shfl_sync(0xffffffffu, v.n, 0)};
}

// Sum of the squared deviations of a piece's first `live` columns; products rounded before they are added, so that all forms of
// a norm (whole pieces, ragged rows) give the same bits whatever the compiler would contract.
__device__ __forceinline__ float piece_sq(float4 v, float mean, int live) {
  const float a = v.x - mean, b = v.y - mean, c = v.z - mean, d = v.w - mean;
  const float aa = __fmul_rn(a, a), bb = __fmul_rn(b, b), cc = __fmul_rn(c, c), dd = __fmul_rn(d, d);
  return (live > 0 ? aa : 0.f) + (live > 1 ? bb : 0.f) + (live > 2 ? cc : 0.f) + (live > 3 ? dd : 0.f);
}

// Subtrahend and factor of a row's norm - layer norm (subtract the mean) or RMS norm (mean of squares) - from the pieces of
// four columns that the threads hold; `n` columns of the row are in this CTA, piece i covers columns 4 (tid + i blockDim).
// Deviations are taken from each thread's own mean and merged pairwise, over the warp, the CTA and the cluster, in an order
// that is the same in every thread.
// FULL: every thread holds whole pieces and the warps' number is a power of two, so that both halves of every merge count the
// same and nothing but means and deviations travels.
template <int NI, bool FULL, class EXCHANGE>
__device__ __forceinline__ float2 row_norm(const float4 (&v)[NI], int n, int W, int kind, float eps, EXCHANGE exchange) {
  const int lane = threadIdx.x & 31;
  if constexpr (FULL) {
    float s = 0.f, q = 0.f;
#pragma unroll
    for (int i = 0; i < NI; ++i) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    float mean = kind == 0 ? s / (4 * NI) : 0.f;                     // an RMS norm merges with zero means
#pragma unroll
    for (int i = 0; i < NI; ++i) q += piece_sq(v[i], mean, 4);
    float half = 2.0f * NI;                // half the number of columns that one side of a merge has
    auto merge_over = [&](int o) {         // merge() of the lower lane's columns and the upper one's, the same in both
      const float m = __shfl_xor_sync(0xffffffffu, mean, o), t = __shfl_xor_sync(0xffffffffu, q, o);
      const bool low = (lane & o) == 0;
      const float d = low ? m - mean : mean - m;
      q = (q + t) + d * d * half;
      mean = (low ? mean : m) + d * 0.5f;
      half *= 2.0f;
    };
    if (kind == 0) {
#pragma unroll
      for (int o = 16; o; o >>= 1) merge_over(o);
    } else {
      q = warp_sum(q);
    }
    const Moments t = exchange(Moments{mean, q, 0.f});
    mean = t.mean;
    q = t.m2;
    for (int o = exchange.warps >> 1; o; o >>= 1) {
      if (kind == 0) merge_over(o);
      else q += __shfl_xor_sync(0xffffffffu, q, o);
    }
    return make_float2(mean, 1.0f / sqrtf(q / W + eps));
  }
  float cnt = 0.f, s = 0.f;              // columns beyond the row hold zeros
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int live = n - 4 * static_cast<int>(threadIdx.x + i * blockDim.x);
    cnt += static_cast<float>(max(0, min(4, live)));
    s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
  }
  const float mean = kind == 0 && cnt > 0.f ? s / cnt : 0.f;         // an RMS norm merges with zero means
  float q = 0.f;
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int live = n - 4 * static_cast<int>(threadIdx.x + i * blockDim.x);
    q += piece_sq(v[i], mean, live);
  }
  Moments t{mean, q, cnt};
  if (kind == 0) t = merge_lanes(t);
  else t.m2 = warp_sum(q);                 // no means to merge
  t = exchange(t);
  if (lane >= exchange.warps) t = {0.f, 0.f, 0.f};
  if (kind == 0) t = merge_lanes(t);
  else t.m2 = warp_sum(t.m2);
  return make_float2(t.mean, 1.0f / sqrtf(t.m2 / W + eps));
}

// What row_norm asks of the threads that share a row: every warp's moments in, lane l gets those of warp l % warps (of `warps`,
// at most 32) out.  One CTA: through shared memory, one barrier.  `slot` holds 3 x 32 floats.
struct BlockExchange {
  float* slot;
  int warps;
  __device__ __forceinline__ Moments operator()(Moments t) const {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
      slot[warp] = t.mean;
      slot[32 + warp] = t.m2;
      slot[64 + warp] = t.n;
    }
    __syncthreads();
    const int w = lane < warps ? lane : lane & (warps - 1);      // the lanes beyond are read where `warps` is a power of two
    return {slot[w], slot[32 + w], slot[64 + w]};
  }
};

// The CTAs of a cluster: every warp sends its moments to all of them, 16 bytes each, and counts on a barrier there; a warp waits for
// its own CTA's copy alone.  (A barrier of the cluster and loads from the peers afterwards: 2000 cycles a norm instead of 1000.)
constexpr int kShare = 8;              // CTAs that share a row
// Rows of more than 16384 columns: beyond this many, a fourth block an SM counts for more than its registers.  20000 columns, three and four
// blocks: 1 row of eight planes 13.7 and 15.5 us, with gate and kept streams 25 and 31; 200 rows 39 and 34, 133 and 118.
constexpr int kLeanRows = 64;
struct RowShare {
  float4 moments[32];
  uint64_t bar;
};
struct ClusterExchange {
  RowShare* sh;
  int rank, warps;
  int* status;
  __device__ __forceinline__ Moments operator()(Moments t) const {
    const int lane = threadIdx.x & 31, at = rank * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (lane < kShare) {
      const uint32_t to = cluster_addr(smem_u32(&sh->moments[at]), lane), bar = cluster_addr(smem_u32(&sh->bar), lane);
      asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                   ::"r"(to), "r"(__float_as_uint(t.mean)), "r"(__float_as_uint(t.m2)), "r"(__float_as_uint(t.n)), "r"(0u), "r"(bar)
                   : "memory");
    }
    __syncwarp();
    if (!mbar_wait(&sh->bar, 0, status, 460))          // reported; what is on its way still lands before the memory changes hands
      for (int i = 0; i < (1 << 20) && !mbar_test_wait(&sh->bar, 0); ++i) {
      }
    const float4 m = sh->moments[lane < warps ? lane : lane & (warps - 1)];
    return {m.x, m.y, m.z};
  }
  // sh->bar counts the stores of all warps; peers may send once the cluster has met after this
  __device__ __forceinline__ static void prepare(RowShare& sh, int warps) {
    mbar_init(&sh.bar, 1);
    mbar_init_fence();
    mbar_expect_tx(&sh.bar, 16 * warps);
  }
};

// Four columns of the sum of a row's routed results, in route order.
__device__ __forceinline__ float4 routed_at4(const ds41_resid_args& p, int r, int col) {
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int k = 0; k < p.y_top; ++k) {
    const int e = p.y_route[r * p.y_top + k];
    if (e < 0) continue;
    const float4 v = proj_at4(p.y, p.y_rows > 0 ? 1ll * e * p.y_rows + r : 1ll * r * p.y_top + k, col);
    s.x += v.x;
    s.y += v.y;
    s.z += v.z;
    s.w += v.w;
  }
  return s;
}

// A thread's pieces of a row of a projection, all under way together: which form it has is asked once, not piece by piece, since a
// test between two loads makes the second one wait for what the first one's value is used for.
template <int NI>
__device__ __forceinline__ void proj_pieces(const ds41_proj& a, long long row, const int (&at)[NI], float4 (&v)[NI]) {
  const long long i0 = row * a.ld + a.col;
  if (a.bf16) {
    uint2 raw[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) raw[i] = *reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(a.data) + i0 + at[i]);
#pragma unroll
    for (int i = 0; i < NI; ++i)
      v[i] = make_float4(__uint_as_float(raw[i].x << 16), __uint_as_float(raw[i].x & 0xffff0000u), __uint_as_float(raw[i].y << 16),
                         __uint_as_float(raw[i].y & 0xffff0000u));
  } else {                                // one fp32 plane
#pragma unroll
    for (int i = 0; i < NI; ++i) v[i] = *reinterpret_cast<const float4*>(static_cast<const float*>(a.data) + i0 + at[i]);
  }
}
// The same of the sum of a row's routed results (bf16 rows, one per route, at most four routes), in route order.
constexpr int kRoutes = 4;
template <int NI>
__device__ __forceinline__ void routed_pieces(const ds41_resid_args& p, int r, const int (&at)[NI], float4 (&v)[NI]) {
  bool on[kRoutes];
  uint2 raw[kRoutes][NI];
#pragma unroll
  for (int k = 0; k < kRoutes; ++k) on[k] = k < p.y_top && p.y_route[r * p.y_top + k] >= 0;
#pragma unroll
  for (int k = 0; k < kRoutes; ++k) {
    const __nv_bfloat16* row = static_cast<const __nv_bfloat16*>(p.y.data) + (1ll * r * p.y_top + k) * p.y.ld + p.y.col;
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (k < p.y_top) raw[k][i] = *reinterpret_cast<const uint2*>(row + at[i]);       // a dropped route's row is there too
  }
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < kRoutes; ++k)
      if (on[k])
        v[i] += make_float4(__uint_as_float(raw[k][i].x << 16), __uint_as_float(raw[k][i].x & 0xffff0000u),
                            __uint_as_float(raw[k][i].y << 16), __uint_as_float(raw[k][i].y & 0xffff0000u));
  }
}

// Many rows: bound by latency, a block's loads and its two chains of merges one after the other.  Rows that fill the threads'
// pieces (FULL) shorten the chain by every test of a column against the row's end, and where their form allows it (TOGETHER, see
// pieces_together) ask for stream, result and gate at once.  Piece by piece, with a test of the projection's form between two loads,
// 2048 rows x 4096 columns took 28 us (plain result), 49 (gated, two norms), 73 (the same with four kept streams) and 54 (four
// routes); together 26, 44, 70 and 26; 953 rows with routes 30 and 16.  Kept streams stay behind the first norm: asked for with the
// rest they cost the registers of a third block an SM (kept streams 82 us).  The forms are kernels of their own: in one they
// spilled, 2048 rows x 1024 columns 9.5 us (7.8 so).  Results of several planes come in passes of few rows, whose blocks need no
// neighbours: those of two pieces take what registers they like (33 rows x 2048, gate and kept streams 8.2 and 7.2 us).
template <typename T, int NI, bool FULL, bool TOGETHER>
__global__ void __launch_bounds__(NI <= 4 ? 256 : 512, NI == 2 && FULL && !TOGETHER ? 1 : 0) resid_step_kernel(ds41_resid_args p) {
  __shared__ float slots[2][96];
  const int r = blockIdx.x, n_warps = blockDim.x >> 5;
  pdl_launch_dependents();
  pdl_wait();
  float4 x[NI];
  int at[NI], live[NI];
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    at[i] = 4 * (threadIdx.x + i * blockDim.x);
    live[i] = FULL ? 4 : p.W - at[i];
    x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (p.tokens != nullptr) {
    const int tok = p.tokens[r];
    const ds41_proj e{p.embed, 0, static_cast<int>(p.embed_ld), 1, 1, 0};
    if (tok >= 0 && tok < p.vocab)
#pragma unroll
      for (int i = 0; i < NI; ++i)
        if (live[i] > 0) x[i] = proj_at4(e, tok, at[i]);
  } else {
    const float* in = p.x_in + r * p.ldx;
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (live[i] > 0) x[i] = *reinterpret_cast<const float4*>(in + at[i]);
  }
  auto clip = [&](float4& v, int i) {         // columns beyond the row hold zeros
    if (FULL) return;
    if (live[i] < 4) v.w = 0.f;
    if (live[i] < 3) v.z = 0.f;
    if (live[i] < 2) v.y = 0.f;
  };
  if (p.y.data != nullptr) {
    float4 y[NI];
    auto gated = [&](float4& v, const float4& g, const float4& b) {
      v.x *= sigmoid_f32(g.x + b.x);
      v.y *= sigmoid_f32(g.y + b.y);
      v.z *= sigmoid_f32(g.z + b.z);
      v.w *= sigmoid_f32(g.w + b.w);
    };
    if constexpr (TOGETHER) {
      if (p.y_route != nullptr) routed_pieces(p, r, at, y);
      else proj_pieces(p.y, r, at, y);
      float4 g[NI];
      if (p.gate.data != nullptr) proj_pieces(p.gate, r, at, g);
      if (p.gate.data != nullptr)
#pragma unroll
        for (int i = 0; i < NI; ++i) gated(y[i], g[i], load4(p.gate_bias + at[i], 4));
    } else {
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        y[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (live[i] > 0) {
          y[i] = p.y_route != nullptr ? routed_at4(p, r, at[i]) : proj_at4(p.y, r, at[i]);
          if (p.gate.data != nullptr) gated(y[i], proj_at4(p.gate, r, at[i]), load4(p.gate_bias + at[i], live[i]));
          clip(y[i], i);
        }
      }
    }
    float2 s = make_float2(0.f, 1.f);
    if (p.post_w != nullptr) s = row_norm<NI, FULL>(y, p.W, p.W, p.post_rms ? 1 : p.norm_kind, p.eps, BlockExchange{slots[0], n_warps});
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (live[i] > 0) {
        const float4 w = p.post_w != nullptr ? load4(p.post_w + at[i], live[i]) : make_float4(1.f, 1.f, 1.f, 1.f);
        x[i].x += (y[i].x - s.x) * s.y * w.x;
        x[i].y += (y[i].y - s.x) * s.y * w.y;
        x[i].z += (y[i].z - s.x) * s.y * w.z;
        x[i].w += (y[i].w - s.x) * s.y * w.w;
      }
  }
#pragma unroll
  for (int i = 0; i < NI; ++i) clip(x[i], i);
  if (p.x_out != nullptr) {
    float* o = p.x_out + r * p.ldx;
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (live[i] > 0) store4(o + at[i], x[i]);
  }
  if (p.mix != nullptr) {
    float4 older[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) older[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* k0 = p.kept + r * p.ldx;
#pragma unroll 4
    for (int j = 0; j < p.n_mix - 1; ++j) {
      const float c = p.mix[j];
#pragma unroll
      for (int i = 0; i < NI; ++i)
        if (live[i] > 0) {
          const float4 k = *reinterpret_cast<const float4*>(k0 + j * p.kept_stride + at[i]);
          older[i].x += c * k.x;
          older[i].y += c * k.y;
          older[i].z += c * k.z;
          older[i].w += c * k.w;
        }
    }
    const float last = p.mix[p.n_mix - 1];    // the newest kept stream is the row this block holds
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      x[i] = make_float4(older[i].x + last * x[i].x, older[i].y + last * x[i].y, older[i].z + last * x[i].z,
                         older[i].w + last * x[i].w);
      clip(x[i], i);
    }
    if (p.x_avg != nullptr) {
      float* o = p.x_avg + r * p.ldx;
#pragma unroll
      for (int i = 0; i < NI; ++i)
        if (live[i] > 0) store4(o + at[i], x[i]);
    }
  }
  if (p.next_w != nullptr) {
    const float2 s = row_norm<NI, FULL>(x, p.W, p.W, p.norm_kind, p.eps, BlockExchange{slots[1], n_warps});
    T* h = static_cast<T*>(p.h) + 1ll * r * p.ldh;
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (live[i] > 0) {
        const float4 w = load4(p.next_w + at[i], live[i]);
        store4(h + at[i], make_float4((x[i].x - s.x) * s.y * w.x, (x[i].y - s.x) * s.y * w.y, (x[i].z - s.x) * s.y * w.z,
                                      (x[i].w - s.x) * s.y * w.w));
      }
  }
  if (p.next_w == nullptr && p.raw_h) {
    T* h = static_cast<T*>(p.h) + 1ll * r * p.ldh;
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (live[i] > 0) store4(h + at[i], x[i]);
  }
}

// A place of a projection whose loads are under way: its planes (up to eight; sixteen would leave room for one CTA beside a GEMM's),
// or the bf16 value.
struct Ahead {
  float4 t[kPlanes];
  __device__ __forceinline__ void ask(const ds41_proj& a, long long row, int col) {
    const long long i = row * a.ld + a.col + col;
    if (a.bf16) t[0] = proj_at4(a, row, col);
    else fetch_planes(t, static_cast<const float*>(a.data) + i, a.plane, a.splits);
  }
  __device__ __forceinline__ float4 get(const ds41_proj& a, long long row, int col) {
    if (a.bf16 || a.splits == 1) return t[0];
    return add_planes(t, static_cast<const float*>(a.data) + row * a.ld + a.col + col, a.plane, a.splits);
  }
};

// A row's routed results again, ids and rows under way together.
__device__ __forceinline__ float4 routed_few4(const ds41_resid_args& p, int r, int col) {
  constexpr int kMost = 8;
  if (p.y_top > kMost || p.y.bf16 || p.y.splits != 1) return routed_at4(p, r, col);
  int e[kMost];
  float4 v[kMost], s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < kMost; ++k) e[k] = k < p.y_top ? p.y_route[r * p.y_top + k] : -1;
  const float* base = static_cast<const float*>(p.y.data) + p.y.col + col;
#pragma unroll
  for (int k = 0; k < kMost; ++k)
    if (e[k] >= 0)
      v[k] = *reinterpret_cast<const float4*>(base + (p.y_rows > 0 ? 1ll * e[k] * p.y_rows + r : 1ll * r * p.y_top + k) * p.y.ld);
#pragma unroll
  for (int k = 0; k < kMost; ++k)
    if (e[k] >= 0) s += v[k];
  return s;
}

// Few rows: a cluster of eight CTAs shares a row, so that its loads do not queue on one SM.  The launch is a chain of latencies:
// weights are read before the wait for the previous kernel, everything else is asked for at once behind it (rows of up to 4096
// columns, a piece of four a thread), and each norm costs one way to the peers.  Inside a graph, one row of 2048 columns with
// kept streams and eight planes of result and gate: 10.3 us with loads plane by plane, divisions in every merge of moments and a
// cluster barrier with loads from the peers behind it, 6.5 so; eight rows without kept streams 5.0 and 4.2.
template <typename T, int NI, bool FULL, int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS) resid_few_kernel(ds41_resid_args p) {
  __shared__ RowShare share[2];
  const int per = ((p.W + kShare - 1) / kShare + 3) / 4 * 4;
  const int part = blockIdx.x % kShare, r = blockIdx.x / kShare, lane = threadIdx.x & 31;
  const int c0 = min(p.W, part * per), n = min(p.W, c0 + per) - c0, warps = kShare * (blockDim.x >> 5);
  if (threadIdx.x == 0) {
    ClusterExchange::prepare(share[0], warps);
    ClusterExchange::prepare(share[1], warps);
  }
  cg::cluster_group::barrier_arrive();
  pdl_launch_dependents();
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), one = make_float4(1.f, 1.f, 1.f, 1.f);
  // More pieces than the registers hold beside their weights: those are read, and the stream stored, where they are needed.  With
  // everything held, 200 rows of 20000 columns took 69 us (plain bf16 result), 95 (gated) and 190 (with kept streams).
  constexpr bool kLean = NI > 2;
  constexpr int kHeld = kLean ? 1 : NI;
  float4 x[NI], y[NI], older[NI], w_next[kHeld], w_post[kHeld], bias[kHeld], stream[kHeld];
  int at[NI], live[NI];
  auto next_at = [&](int i) { return p.next_w != nullptr && live[i] > 0 ? load4(p.next_w + at[i], live[i]) : zero; };
  auto post_at = [&](int i) { return p.post_w != nullptr && live[i] > 0 ? load4(p.post_w + at[i], live[i]) : one; };
  auto bias_at = [&](int i) { return p.gate.data != nullptr && live[i] > 0 ? load4(p.gate_bias + at[i], live[i]) : zero; };
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int c = 4 * (threadIdx.x + i * blockDim.x);
    live[i] = FULL ? 4 : n - c;
    at[i] = c0 + c;
    x[i] = y[i] = older[i] = zero;
    if constexpr (!kLean) {
      w_next[i] = next_at(i);
      w_post[i] = post_at(i);
      bias[i] = bias_at(i);
    }
  }
  const int n_old = p.mix != nullptr ? p.n_mix - 1 : 0;
  const float mix_lane = lane <= n_old && p.mix != nullptr ? p.mix[lane] : 0.f;
  auto weight = [&](int j) { return j < 32 ? __shfl_sync(0xffffffffu, mix_lane, j) : p.mix[j]; };
  cg::cluster_group::barrier_wait();
  pdl_wait();
  // ---- loads
  const float* kept = p.kept + r * p.ldx;
  const bool plain = p.y.data != nullptr && p.y_route == nullptr;
  constexpr bool kAhead = NI == 1;         // one piece a thread: everything is under way before the first sum
  Ahead ya, ga;
  float4 ka[kPlanes];
  if (p.tokens != nullptr) {
    const int tok = p.tokens[r];
    const ds41_proj e{p.embed, 0, static_cast<int>(p.embed_ld), 1, 1, 0};
    if (tok >= 0 && tok < p.vocab)
#pragma unroll
      for (int i = 0; i < NI; ++i)
        if (live[i] > 0) x[i] = proj_at4(e, tok, at[i]);
  } else {
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (live[i] > 0) x[i] = *reinterpret_cast<const float4*>(p.x_in + r * p.ldx + at[i]);
  }
  if (kAhead && live[0] > 0) {
    if (plain) ya.ask(p.y, r, at[0]);
    if (p.y.data != nullptr && p.gate.data != nullptr) ga.ask(p.gate, r, at[0]);
    fetch_planes(ka, kept + at[0], p.kept_stride, n_old);
  }
  if (p.y.data != nullptr && p.y_route != nullptr)
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (live[i] > 0) y[i] = kLean ? routed_at4(p, r, at[i]) : routed_few4(p, r, at[i]);
  // ---- the weighted sum of the older kept streams
  auto add_old = [&](int i, float c, float4 k) {
    older[i].x += c * k.x;
    older[i].y += c * k.y;
    older[i].z += c * k.z;
    older[i].w += c * k.w;
  };
  if constexpr (kAhead) {
    for (int j0 = 0; j0 < n_old; j0 += kPlanes) {
      if (j0 > 0 && live[0] > 0) fetch_planes(ka, kept + j0 * p.kept_stride + at[0], p.kept_stride, n_old - j0);
#pragma unroll
      for (int u = 0; u < kPlanes; ++u)
        if (j0 + u < n_old) {
          const float c = weight(j0 + u);
          if (live[0] > 0) add_old(0, c, ka[u]);
        }
    }
  } else {
#pragma unroll 4
    for (int j = 0; j < n_old; ++j) {
      const float c = weight(j);
#pragma unroll
      for (int i = 0; i < NI; ++i)
        if (live[i] > 0) add_old(i, c, *reinterpret_cast<const float4*>(kept + j * p.kept_stride + at[i]));
    }
  }
  auto clip = [&](float4& v, int i) {         // columns beyond the row hold zeros
    if (FULL) return;
    if (live[i] < 4) v.w = 0.f;
    if (live[i] < 3) v.z = 0.f;
    if (live[i] < 2) v.y = 0.f;
  };
  // ---- the sublayer's result
  if (p.y.data != nullptr) {
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (live[i] > 0) {
        if (plain) y[i] = kAhead ? ya.get(p.y, r, at[i]) : kLean ? proj_at4(p.y, r, at[i]) : few_at4(p.y, r, at[i]);
        if (p.gate.data != nullptr) {
          const float4 g = kAhead ? ga.get(p.gate, r, at[i]) : kLean ? proj_at4(p.gate, r, at[i]) : few_at4(p.gate, r, at[i]);
          const float4 b = kLean ? bias_at(i) : bias[i % kHeld];
          y[i].x *= sigmoid_f32(g.x + b.x);
          y[i].y *= sigmoid_f32(g.y + b.y);
          y[i].z *= sigmoid_f32(g.z + b.z);
          y[i].w *= sigmoid_f32(g.w + b.w);
        }
        clip(y[i], i);
      }
    float2 s = make_float2(0.f, 1.f);
    if (p.post_w != nullptr)
      s = row_norm<NI, FULL>(y, n, p.W, p.post_rms ? 1 : p.norm_kind, p.eps, ClusterExchange{&share[0], part, warps, p.status});
#pragma unroll
    for (int i = 0; i < NI; ++i)
      if (live[i] > 0) {
        const float4 w = kLean ? post_at(i) : w_post[i % kHeld];
        x[i].x += (y[i].x - s.x) * s.y * w.x;
        x[i].y += (y[i].y - s.x) * s.y * w.y;
        x[i].z += (y[i].z - s.x) * s.y * w.z;
        x[i].w += (y[i].w - s.x) * s.y * w.w;
      }
  }
  const float last = p.mix != nullptr ? weight(n_old) : 0.f;      // the newest kept stream is the row this block holds
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    clip(x[i], i);
    if constexpr (!kLean) stream[i] = x[i];
    else if (p.x_out != nullptr && live[i] > 0) store4(p.x_out + r * p.ldx + at[i], x[i]);
    if (p.mix != nullptr) {                  // from here on x is what the next sublayer sees
      x[i] = make_float4(older[i].x + last * x[i].x, older[i].y + last * x[i].y, older[i].z + last * x[i].z,
                         older[i].w + last * x[i].w);
      clip(x[i], i);
    }
  }
  float2 s = make_float2(0.f, 1.f);
  if (p.next_w != nullptr) s = row_norm<NI, FULL>(x, n, p.W, p.norm_kind, p.eps, ClusterExchange{&share[1], part, warps, p.status});
  cg::cluster_group::barrier_arrive();
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    if (live[i] <= 0) continue;
    if (!kLean && p.x_out != nullptr) store4(p.x_out + r * p.ldx + at[i], stream[i % kHeld]);
    if (p.mix != nullptr && p.x_avg != nullptr) store4(p.x_avg + r * p.ldx + at[i], x[i]);
    T* h = static_cast<T*>(p.h) + 1ll * r * p.ldh + at[i];
    if (p.next_w != nullptr) {
      const float4 w = kLean ? next_at(i) : w_next[i % kHeld];
      store4(h, make_float4((x[i].x - s.x) * s.y * w.x, (x[i].y - s.x) * s.y * w.y, (x[i].z - s.x) * s.y * w.z,
                            (x[i].w - s.x) * s.y * w.w));
    } else if (p.raw_h) {
      store4(h, x[i]);
    }
  }
  cg::cluster_group::barrier_wait();           // no CTA leaves while a peer may still send to it
}

template <typename T>
__global__ void __launch_bounds__(512) polynorm_kernel(ds41_proj z, const float* coef, int ff, int ld_out, float eps,
                                                       T* out) {
  extern __shared__ float zrow[];
  __shared__ float red[3][32];
  const int r = blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  float s2 = 0.f, s4 = 0.f, s6 = 0.f;
  auto add = [&](float v) {
    const float q = v * v;
    s2 += q;
    s4 += q * q;
    s6 += q * q * q;
  };
#pragma unroll 4
  for (int i = 4 * threadIdx.x; i < ff; i += 4 * blockDim.x) {
    float4 v = proj_at4(z, r, i);
    if (i + 3 >= ff) v.w = 0.f;            // columns beyond ff add nothing to the sums
    if (i + 2 >= ff) v.z = 0.f;
    if (i + 1 >= ff) v.y = 0.f;
    *reinterpret_cast<float4*>(zrow + i) = v;
    add(v.x);
    add(v.y);
    add(v.z);
    add(v.w);
  }
  // the three sums over the block behind one barrier; every warp adds the warps' shares itself (2048 rows of 11008 columns: 34.3
  // us with one block-wide sum after the other, 32.1 so; 1 row 5.3 and 4.7)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  s2 = warp_sum(s2);
  s4 = warp_sum(s4);
  s6 = warp_sum(s6);
  if (lane == 0) {
    red[0][warp] = s2;
    red[1][warp] = s4;
    red[2][warp] = s6;
  }
  __syncthreads();
  s2 = warp_sum(lane < n_warps ? red[0][lane] : 0.f);
  s4 = warp_sum(lane < n_warps ? red[1][lane] : 0.f);
  s6 = warp_sum(lane < n_warps ? red[2][lane] : 0.f);
  const float a = coef[0] / sqrtf(s2 / ff + eps), b = coef[1] / sqrtf(s4 / ff + eps), c = coef[2] / sqrtf(s6 / ff + eps);
  const float e = coef[3];
  auto act = [&](float v) { return ((c * v + b) * v + a) * v + e; };
  for (int i = 4 * threadIdx.x; i < ff; i += 4 * blockDim.x) {
    const float4 v = *reinterpret_cast<const float4*>(zrow + i);
    store4(out + 1ll * r * ld_out + i, make_float4(act(v.x), act(v.y), act(v.z), act(v.w)));
  }
}

template <typename T, bool FEW>
__global__ void __launch_bounds__(256) gate_mul_kernel(ds41_proj y, ds41_proj gate, int n, T* out, int ld_out) {
  const int r = blockIdx.y, i = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  pdl_launch_dependents();
  pdl_wait();
  if (i >= n) return;
  const float4 v = at4<FEW>(y, r, i), g = at4<FEW>(gate, r, i);
  store4(out + 1ll * r * ld_out + i, make_float4(v.x * sigmoid_f32(g.x), v.y * sigmoid_f32(g.y), v.z * sigmoid_f32(g.z),
                                                 v.w * sigmoid_f32(g.w)));
}

// one block per (row, head); columns [width, stride) of a head are padding and are written as zeros
template <typename T, bool FEW>
__global__ void __launch_bounds__(128) head_norm_gate_kernel(const float* o, int ld_o, ds41_proj gate, const float* w,
                                                             int width, int stride, float eps, T* out, int ld_out) {
  __shared__ float red[4];
  const int h = blockIdx.x, r = blockIdx.y;
  pdl_launch_dependents();
  pdl_wait();
  const float* src = o + 1ll * r * ld_o + h * stride;
  T* dst = out + 1ll * r * ld_out + h * stride;
  float q = 0.f;
  float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), g0 = v0, w0 = v0;       // the thread's first piece stays in registers
  for (int i = 4 * threadIdx.x; i < stride; i += 4 * blockDim.x) {
    const float4 v = load4(src + i, width - i);
    if (i < 4 * static_cast<int>(blockDim.x)) {
      v0 = v;
      g0 = at4<FEW>(gate, r, h * stride + i);
      w0 = load4(w + h * stride + i, width - i);
    }
    q += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  q = warp_sum(q);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = q;
  __syncthreads();
  q = 0.f;
  for (int i = 0; i < static_cast<int>(blockDim.x >> 5); ++i) q += red[i];
  const float s = 1.0f / sqrtf(q / width + eps);
  for (int i = 4 * threadIdx.x; i < stride; i += 4 * blockDim.x) {
    const bool first = i < 4 * static_cast<int>(blockDim.x);
    const float4 v = first ? v0 : load4(src + i, width - i), ww = first ? w0 : load4(w + h * stride + i, width - i);
    const float4 g = first ? g0 : proj_at4(gate, r, h * stride + i);
    store4(dst + i, make_float4(i < width ? v.x * s * ww.x * sigmoid_f32(g.x) : 0.f,
                                i + 1 < width ? v.y * s * ww.y * sigmoid_f32(g.y) : 0.f,
                                i + 2 < width ? v.z * s * ww.z * sigmoid_f32(g.z) : 0.f,
                                i + 3 < width ? v.w * s * ww.w * sigmoid_f32(g.w) : 0.f));
  }
}

// many (row, head) pairs of at most 512 columns: one warp each
template <typename T>
__global__ void __launch_bounds__(256) head_norm_gate_warp_kernel(const float* o, int ld_o, ds41_proj gate, const float* w,
                                                                  int items, int heads, int width, int stride, float eps,
                                                                  T* out, int ld_out) {
  const int item = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_launch_dependents();
  pdl_wait();
  if (item >= items) return;
  const int r = item / heads, h = item - r * heads;
  const float* src = o + 1ll * r * ld_o + h * stride;
  T* dst = out + 1ll * r * ld_out + h * stride;
  float4 v[4], g[4];
  float q = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = 4 * (lane + 32 * k);
    v[k] = g[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < stride) {
      v[k] = load4(src + i, width - i);
      g[k] = proj_at4(gate, r, h * stride + i);
    }
    q += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
  }
  const float s = 1.0f / sqrtf(warp_sum(q) / width + eps);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = 4 * (lane + 32 * k);
    if (i >= stride) break;
    const float4 ww = load4(w + h * stride + i, width - i);
    store4(dst + i, make_float4(i < width ? v[k].x * s * ww.x * sigmoid_f32(g[k].x) : 0.f,
                                i + 1 < width ? v[k].y * s * ww.y * sigmoid_f32(g[k].y) : 0.f,
                                i + 2 < width ? v[k].z * s * ww.z * sigmoid_f32(g[k].z) : 0.f,
                                i + 3 < width ? v[k].w * s * ww.w * sigmoid_f32(g[k].w) : 0.f));
  }
}

// one block per row; columns [n, ld_out) are written as zeros
template <typename T, bool FEW>
__global__ void __launch_bounds__(128) side_act_kernel(ds41_proj z, const int* tokens, const __nv_bfloat16* embed,
                                                       long long embed_ld, int col, int vocab, int n, T* out, int ld_out) {
  const int r = blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  const int tok = tokens[r];
  const bool known = tok >= 0 && tok < vocab;
  for (int j = threadIdx.x; j < ld_out; j += blockDim.x) {
    float v = 0.f;
    if (j < n) {
      const float a = at1<FEW>(z, r, j);
      const float e = known ? __bfloat162float(embed[tok * embed_ld + col + j]) : 0.f;
      v = 0.5f * a * (1.0f + tanhf(0.7978845608028654f * (a + 0.044715f * a * a * a))) * e;
    }
    out[1ll * r * ld_out + j] = from_f32<T>(v);
  }
}

__global__ void __launch_bounds__(256) softcap_kernel(float* x, long long n, float cap) {
  const long long i = 1ll * blockIdx.x * blockDim.x + threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  if (i < n) x[i] = cap * tanhf(x[i] / cap);
}

template <typename T>
__global__ void __launch_bounds__(256) gather_rows_kernel(const T* src, int ld, const int* index, int n_src, int W, T* dst) {
  const int r = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  if (i >= W) return;
  const int s = index[r];
  dst[1ll * r * ld + i] = s >= 0 && s < n_src ? src[1ll * s * ld + i] : from_f32<T>(0.f);
}

// Can result and gate be asked for in whole pieces: bf16 or one plane, or up to four routes of bf16 rows?  (Not for one piece a thread,
// which has nothing to ask for together.)
static bool pieces_together(const ds41_resid_args& a) {
  auto one = [](const ds41_proj& p) { return p.bf16 || p.splits == 1; };
  const bool y = a.y_route != nullptr ? a.y.bf16 && a.y_rows == 0 && a.y_top <= kRoutes : one(a.y);
  return a.y.data != nullptr && y && (a.gate.data == nullptr || one(a.gate));
}

// FULL: a row fills the pieces of the threads that share it, whose warps' number is a power of two
template <typename T, bool FEW, int NI>
static cudaError_t launch_resid_ni(const ds41_resid_args& a, int threads, cudaStream_t st) {
  const bool even = (threads & (threads - 1)) == 0;
  if constexpr (!FEW) {
    if (even && a.W == 4 * NI * threads) {
      if constexpr (NI > 1)
        if (pieces_together(a)) return launch_pdl(resid_step_kernel<T, NI, true, true>, dim3(a.rows), dim3(threads), 0, st, a);
      return launch_pdl(resid_step_kernel<T, NI, true, false>, dim3(a.rows), dim3(threads), 0, st, a);
    }
    return launch_pdl(resid_step_kernel<T, NI, false, false>, dim3(a.rows), dim3(threads), 0, st, a);
  } else {
    auto launch = [&](auto full, auto blocks) {
      return launch_pdl_cluster(resid_few_kernel<T, NI, decltype(full)::value, decltype(blocks)::value>, dim3(a.rows * kShare), dim3(threads),
                                kShare, 0, st, a);
    };
    auto pick = [&](auto full) {
      if constexpr (NI < 8) return launch(full, std::integral_constant<int, 0>{});
      else return a.rows > kLeanRows ? launch(full, std::integral_constant<int, 4>{}) : launch(full, std::integral_constant<int, 3>{});
    };
    return even && a.W == kShare * 4 * NI * threads ? pick(std::true_type{}) : pick(std::false_type{});
  }
}

template <typename T, bool FEW>
static cudaError_t launch_resid(const ds41_resid_args& a, cudaStream_t st) {
  const int ctas = FEW ? kShare : 1, pieces = ((a.W + ctas - 1) / ctas + 3) / 4;
  const auto width = [&](int ni) { return ((pieces + ni - 1) / ni + 31) / 32 * 32; };
  constexpr int kMost = FEW ? 128 : 256;            // the moments of a cluster's warps fit one warp
  if (width(1) <= kMost) return launch_resid_ni<T, FEW, 1>(a, width(1), st);
  if (width(2) <= kMost) return launch_resid_ni<T, FEW, 2>(a, width(2), st);
  if (width(4) <= kMost) return launch_resid_ni<T, FEW, 4>(a, width(4), st);
  if (width(8) <= (FEW ? 128 : 512)) return launch_resid_ni<T, FEW, 8>(a, width(8), st);
  return cudaErrorInvalidValue;
}

}  // namespace ds41

using namespace ds41;

extern "C" int ds41_resid_step(const ds41_resid_args* a, void* stream) {
  if (a == nullptr || a->rows <= 0 || a->W <= 0 || a->ldx < a->W) return cudaErrorInvalidValue;
  if (a->tokens != nullptr ? (a->embed == nullptr || a->embed_ld < a->W || a->vocab <= 0) : a->x_in == nullptr)
    return cudaErrorInvalidValue;
  if (a->y.data != nullptr && !proj_ok(a->y)) return cudaErrorInvalidValue;
  if (a->gate.data != nullptr && (!proj_ok(a->gate) || a->gate_bias == nullptr)) return cudaErrorInvalidValue;
  if (a->mix != nullptr && (a->n_mix < 1 || (a->n_mix > 1 && a->kept == nullptr))) return cudaErrorInvalidValue;
  if (a->y_route != nullptr && (a->y.data == nullptr || a->y_top <= 0 || a->y_rows < 0)) return cudaErrorInvalidValue;
  if ((a->next_w != nullptr || a->raw_h) && (a->h == nullptr || a->ldh < a->W || (a->ldh & 3))) return cudaErrorInvalidValue;
  // rows are walked in pieces of four columns
  if ((a->ldx & 3) || (a->kept_stride & 3) || (a->tokens != nullptr && (a->embed_ld & 3)) ||
      (a->y.data != nullptr && !proj_vec4(a->y)) || (a->gate.data != nullptr && !proj_vec4(a->gate)))
    return cudaErrorInvalidValue;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // few rows: a cluster of eight CTAs shares a row, so that its loads do not queue on one SM
  const bool wide = (a->rows <= 32 && a->W >= 1024) || a->W > 16384;
  if (a->f32) return wide ? launch_resid<float, true>(*a, st) : launch_resid<float, false>(*a, st);
  return wide ? launch_resid<__nv_bfloat16, true>(*a, st) : launch_resid<__nv_bfloat16, false>(*a, st);
}

template <typename T>
static int launch_polynorm(const ds41_proj& z, const float* coef, int rows, int ff, int ld_out, float eps, void* out,
                           cudaStream_t st) {
  const size_t smem = (1ull * ff + 3) / 4 * 16;
  static size_t allowed = 48 * 1024 - 512;
  if (smem > allowed) {
    if (smem > 226 * 1024) return cudaErrorInvalidValue;
    const cudaError_t e = cudaFuncSetAttribute(polynorm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    allowed = smem;
  }
  return launch_pdl(polynorm_kernel<T>, dim3(rows), dim3(ff >= 2048 ? 512 : 256), smem, st, z, coef, ff, ld_out, eps,
                    static_cast<T*>(out));
}

extern "C" int ds41_polynorm(const ds41_proj* z, const float* coef, int rows, int ff, float eps, void* out, int ld_out,
                             int f32, void* stream) {
  if (z == nullptr || !proj_ok(*z) || !proj_vec4(*z) || coef == nullptr || out == nullptr || rows <= 0 || ff <= 0 ||
      ld_out < ff || (ld_out & 3) || z->ld < z->col + (ff + 3) / 4 * 4)
    return cudaErrorInvalidValue;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return f32 ? launch_polynorm<float>(*z, coef, rows, ff, ld_out, eps, out, st)
             : launch_polynorm<__nv_bfloat16>(*z, coef, rows, ff, ld_out, eps, out, st);
}

extern "C" int ds41_gate_mul(const ds41_proj* y, const ds41_proj* gate, int rows, int n, void* out, int ld_out, int f32,
                             void* stream) {
  if (y == nullptr || gate == nullptr || !proj_ok(*y) || !proj_ok(*gate) || out == nullptr || rows <= 0 || n <= 0 ||
      ld_out < n || rows > 65535 || (n & 3) || (ld_out & 3) || !proj_vec4(*y) || !proj_vec4(*gate))
    return cudaErrorInvalidValue;
  const dim3 grid((n + 1023) / 1024, rows);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // 4096 columns, us with planes together / one after the other: 64 rows (256 blocks) of four 2.7 / 3.1, 200 rows (800) 4.0 / 3.6; 2048 rows
  // of one 16.6 / 12.8
  const long long blocks = 1ll * grid.x * rows;
  const bool few = planes_together(*y, blocks, 4 * sm_count()) || planes_together(*gate, blocks, 4 * sm_count());
  auto launch = [&](auto kernel, auto* o) { return launch_pdl(kernel, grid, dim3(256), 0, st, *y, *gate, n, o, ld_out); };
  if (f32) return launch(few ? gate_mul_kernel<float, true> : gate_mul_kernel<float, false>, static_cast<float*>(out));
  return launch(few ? gate_mul_kernel<__nv_bfloat16, true> : gate_mul_kernel<__nv_bfloat16, false>, static_cast<__nv_bfloat16*>(out));
}

extern "C" int ds41_head_norm_gate(const float* o, int ld_o, const ds41_proj* gate, const float* w, int rows, int heads,
                                   int width, int stride, float eps, void* out, int ld_out, int f32, void* stream) {
  if (o == nullptr || gate == nullptr || !proj_ok(*gate) || w == nullptr || out == nullptr || rows <= 0 || heads <= 0 ||
      width <= 0 || stride < width || (stride & 3) || ld_o < heads * stride || (ld_o & 3) || ld_out < heads * stride ||
      (ld_out & 3) || !proj_vec4(*gate) || rows > 65535)
    return cudaErrorInvalidValue;
  const dim3 grid(heads, rows), block(stride >= 512 ? 128 : (stride + 127) / 128 * 32);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (stride <= 512 && rows * heads >= 1024) {
    const dim3 warps((rows * heads + 7) / 8);
    if (f32)
      return launch_pdl(head_norm_gate_warp_kernel<float>, warps, dim3(256), 0, st, o, ld_o, *gate, w, rows * heads, heads,
                        width, stride, eps, static_cast<float*>(out), ld_out);
    return launch_pdl(head_norm_gate_warp_kernel<__nv_bfloat16>, warps, dim3(256), 0, st, o, ld_o, *gate, w, rows * heads,
                      heads, width, stride, eps, static_cast<__nv_bfloat16*>(out), ld_out);
  }
  // heads of 256, us with planes together / one after the other: 8 rows of 4096 (128 blocks) of four 2.3 / 2.4, of eight 2.4 / 2.7; 32 rows
  // (512) of four 2.8 / 2.6, of one 2.4 / 2.2
  const bool few = planes_together(*gate, 1ll * rows * heads, 2 * sm_count());
  auto launch = [&](auto kernel, auto* x) { return launch_pdl(kernel, grid, block, 0, st, o, ld_o, *gate, w, width, stride, eps, x, ld_out); };
  if (f32) return launch(few ? head_norm_gate_kernel<float, true> : head_norm_gate_kernel<float, false>, static_cast<float*>(out));
  return launch(few ? head_norm_gate_kernel<__nv_bfloat16, true> : head_norm_gate_kernel<__nv_bfloat16, false>,
                static_cast<__nv_bfloat16*>(out));
}

extern "C" int ds41_side_act(const ds41_proj* z, const int* tokens, const void* embed, long long embed_ld, int col, int vocab,
                             int rows, int n, void* out, int ld_out, int f32, void* stream) {
  if (z == nullptr || !proj_ok(*z) || tokens == nullptr || embed == nullptr || out == nullptr || rows <= 0 || n <= 0 ||
      ld_out < n || col < 0 || embed_ld < col + n || vocab <= 0 || z->ld < z->col + n)
    return cudaErrorInvalidValue;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __nv_bfloat16* e = static_cast<const __nv_bfloat16*>(embed);
  // 256 columns, us with planes together / one after the other: 1 row of two 1.5 / 1.7, 200 rows of four 2.0 / 2.5, 2048 rows of two 4.1 / 3.7
  const bool few = planes_together(*z, rows, 4 * sm_count(), 2);
  auto launch = [&](auto kernel, auto* o) { return launch_pdl(kernel, dim3(rows), dim3(128), 0, st, *z, tokens, e, embed_ld, col, vocab, n, o, ld_out); };
  if (f32) return launch(few ? side_act_kernel<float, true> : side_act_kernel<float, false>, static_cast<float*>(out));
  return launch(few ? side_act_kernel<__nv_bfloat16, true> : side_act_kernel<__nv_bfloat16, false>, static_cast<__nv_bfloat16*>(out));
}

extern "C" int ds41_softcap_rows(float* x, long long n, float cap, void* stream) {
  if (x == nullptr || n <= 0 || !(cap > 0.f) || (n + 255) / 256 > 0x7fffffffll) return cudaErrorInvalidValue;
  return launch_pdl(softcap_kernel, dim3(static_cast<unsigned>((n + 255) / 256)), dim3(256), 0,
                    static_cast<cudaStream_t>(stream), x, n, cap);
}

extern "C" int ds41_gather_rows(const void* src, int ld, const int* index, int n_src, int rows, int W, void* dst, int f32,
                                void* stream) {
  if (src == nullptr || index == nullptr || dst == nullptr || rows <= 0 || W <= 0 || ld < W || rows > 65535)
    return cudaErrorInvalidValue;
  const dim3 grid((W + 255) / 256, rows);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (f32)
    return launch_pdl(gather_rows_kernel<float>, grid, dim3(256), 0, st, static_cast<const float*>(src), ld, index, n_src,
                      W, static_cast<float*>(dst));
  return launch_pdl(gather_rows_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, static_cast<const __nv_bfloat16*>(src), ld,
                    index, n_src, W, static_cast<__nv_bfloat16*>(dst));
}
