// Vocabulary-head epilogues: masked greedy argmax, cross-shard merge, speculative accept.
//
//  argmax_rows   : per row, (max logit, lowest token id) over this rank's vocabulary shard under an optional
//                  packed allow-mask (bit set = allowed), non-finite logits reported through a status word
//                  (greedy contract of native/cuda/kernels/v41_sampling_gpu.cu:303-323)
//  argmax_merge  : deterministic merge of the per-shard candidates (highest value, lowest id)
//                  (native/include/ds41rt_v41_dspark.h:21-34)
//  spec_accept   : accept-prefix rule of speculative verification: draft j is accepted while it equals the
//                  target's choice after draft j-1; emits accepted count and the tokens to emit
//                  (rust/crates/ds41rt-core/src/dspark_verify.rs:18-52)
#include <cooperative_groups.h>

#include "ds41_api.h"
#include "ds41_launch.cuh"
#include "ds41_ptx.cuh"

namespace ds41 {

namespace cg = cooperative_groups;

struct ArgmaxParams {
  const float* logits;    // [rows][ld]
  long long ld;
  int vocab_local, vocab_offset;
  const uint32_t* mask;   // optional [rows][mask_words] over the GLOBAL vocabulary
  int mask_words;
  float* best_val;        // [rows]
  int* best_idx;          // [rows] global token id
  int* row_status;        // optional [rows]: 1 = non-finite logit seen, 2 = no allowed candidate
};

// Where rows are long and few, a cluster of eight CTAs shares one: one CTA keeps too few loads in flight for half a megabyte.
// Short rows do not pay for the cluster and many rows fill the GPU by themselves.  us, one CTA of 1024 threads / a cluster of
// eight of 512: 4096 columns 1 row 2.2 / 2.5, 128 rows 3.0 / 8.8; 32000 columns 16 rows 4.4 / 3.3, 64 rows 5.5 / 6.7; 129280
// columns 1 row 11.1 / 3.8, 128 rows 19.5 / 16.7, 300 rows 38.0 / 39.6; 262144 columns 128 rows 40.1 / 30.2, 1024 rows 164 / 198.
constexpr int kArgmaxCtas = 8;
static bool argmax_in_cluster(int rows, int vocab) { return vocab >= 16384 && rows <= 128 && rows <= vocab / 1024; }

template <int CTAS, int THREADS, int DEEP>                 // every thread has DEEP 16-byte loads in flight
__global__ void __launch_bounds__(THREADS) argmax_rows_kernel(ArgmaxParams p) {
  __shared__ float wv[THREADS / 32];
  __shared__ int wi[THREADS / 32];
  __shared__ int bad;
  __shared__ float cta_v;
  __shared__ int cta_i;
  const int r = blockIdx.x / CTAS, part = blockIdx.x % CTAS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_launch_dependents();
  pdl_wait();
  if (tid == 0) bad = 0;
  __syncthreads();
  float v = -INFINITY;
  int idx = 0x7fffffff;
  int nonfinite = 0;
  const float* row = p.logits + 1ll * r * p.ld;
  const uint32_t* mrow = p.mask != nullptr ? p.mask + 1ll * r * p.mask_words : nullptr;
  auto take = [&](int i, float x) {
    const int tok = p.vocab_offset + i;
    if (!isfinite(x)) nonfinite = 1;
    bool ok = true;
    if (mrow != nullptr) ok = (mrow[tok >> 5] >> (tok & 31)) & 1u;
    if (ok && (x > v || (x == v && tok < idx))) { v = x; idx = tok; }
  };
  const int per = CTAS == 1 ? p.vocab_local : ((p.vocab_local + CTAS - 1) / CTAS + 3) / 4 * 4;       // whole 16-byte pieces
  const int i0 = min(p.vocab_local, part * per), i1 = min(p.vocab_local, i0 + per);
  int i = i0 + tid;
  if ((p.ld & 3) == 0 && (reinterpret_cast<uintptr_t>(p.logits) & 15) == 0) {
    const int g1 = i1 >> 2;
    for (int g0 = (i0 >> 2) + tid; g0 < g1; g0 += THREADS * DEEP) {
      float4 a[DEEP];
      a[0] = *reinterpret_cast<const float4*>(row + 4 * g0);
#pragma unroll
      for (int u = 1; u < DEEP; ++u)
        if (g0 + u * THREADS < g1) a[u] = *reinterpret_cast<const float4*>(row + 4 * (g0 + u * THREADS));
#pragma unroll
      for (int u = 0; u < DEEP; ++u) {
        const int g = g0 + u * THREADS;
        if (g < g1) { take(4 * g, a[u].x); take(4 * g + 1, a[u].y); take(4 * g + 2, a[u].z); take(4 * g + 3, a[u].w); }
      }
    }
    i = max(i0, 4 * g1) + tid;
  }
  for (; i < i1; i += THREADS) take(i, row[i]);
  if (nonfinite) bad = 1;
  auto better = [&](float ov, int oi) {
    if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
  };
  auto better_of_warp = [&]() {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, v, o);
      const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
      better(ov, oi);
    }
  };
  auto finish = [&](int any_bad) {
    p.best_val[r] = v;
    p.best_idx[r] = idx == 0x7fffffff ? -1 : idx;
    if (p.row_status != nullptr) p.row_status[r] = any_bad ? 1 : (idx == 0x7fffffff ? 2 : 0);
  };
  better_of_warp();
  if (lane == 0) { wv[warp] = v; wi[warp] = idx; }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < THREADS / 32; ++w) better(wv[w], wi[w]);
    if (CTAS == 1) finish(bad);
    cta_v = v;
    cta_i = idx;
  }
  if constexpr (CTAS > 1) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (part == 0 && warp == 0) {
      int any_bad = 0;
      v = -INFINITY;
      idx = 0x7fffffff;
      if (lane < CTAS) {
        v = *cluster.map_shared_rank(&cta_v, lane);
        idx = *cluster.map_shared_rank(&cta_i, lane);
        any_bad = *cluster.map_shared_rank(&bad, lane);
      }
      any_bad = __any_sync(0xffffffffu, any_bad);
      better_of_warp();
      if (lane == 0) finish(any_bad);
    }
    cluster.sync();            // the first CTA may still read the others' shared memory
  }
}

// candidates from `n_ranks` shards: vals[k][rows], idxs[k][rows] (pointer tables, possibly peer memory)
struct MergeArgs {
  const float* vals[8];
  const int* idxs[8];
  int n_ranks, rows;
  int* out;     // [rows]
  const uint32_t* const* wait_flags;   // optional device array of n_ranks flag pointers
  const uint32_t* wait_epoch;
  int* status;
};
__global__ void argmax_merge_kernel(MergeArgs p) {
  pdl_launch_dependents();
  pdl_wait();
  if (p.wait_flags != nullptr && p.n_ranks > 1) {
    if (threadIdx.x < p.n_ranks) flag_wait_ge(p.wait_flags[threadIdx.x], *p.wait_epoch, p.status, 500 + threadIdx.x);
    __syncthreads();
  }
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= p.rows) return;
  float v = -INFINITY;
  int idx = -1;
  // every rank's candidate is requested before the first comparison: a peer load takes a few microseconds
  for (int k0 = 0; k0 < p.n_ranks; k0 += 8) {
    float ovs[8];
    int ois[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      ovs[u] = -INFINITY;
      ois[u] = -1;
      if (k0 + u < p.n_ranks) { ovs[u] = p.vals[k0 + u][r]; ois[u] = p.idxs[k0 + u][r]; }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float ov = ovs[u];
      const int oi = ois[u];
      if (oi >= 0 && (idx < 0 || ov > v || (ov == v && oi < idx))) { v = ov; idx = oi; }
    }
  }
  p.out[r] = idx;
}

// Verification chunk of request q occupies rows [first[q], first[q] + n[q]): row 0 carries the anchor token,
// row j the j-th draft.  chosen[row] is the target's token AFTER consuming that row's input.
// accepted[q] = number of drafts accepted; emit[q][0..accepted] = chosen tokens of rows 0..accepted.
struct AcceptParams {
  const int* inputs;    // [rows] token fed at each row
  const int* chosen;    // [rows]
  const int* first;     // [reqs]
  const int* count;     // [reqs]
  int reqs, max_emit, eos;
  int* accepted;        // [reqs]
  int* emit;            // [reqs][max_emit]
  int* n_emit;          // [reqs]
};
__global__ void spec_accept_kernel(AcceptParams p) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  if (q >= p.reqs) return;
  const int f = p.first[q], n = p.count[q];
  int acc = 0;
  int emitted = 0;
  for (int j = 0; j < n; ++j) {
    const int tok = p.chosen[f + j];
    if (emitted < p.max_emit) p.emit[q * p.max_emit + emitted] = tok;
    ++emitted;
    if (tok == p.eos) break;                                  // stop token ends the chunk
    if (j + 1 < n && p.inputs[f + j + 1] == tok) ++acc;       // next draft matches -> keep going
    else break;
  }
  p.accepted[q] = acc;
  p.n_emit[q] = min(emitted, p.max_emit);
}

// Device-side feedback for back-to-back decode steps: next input token = chosen token, position + 1.
__global__ void decode_feedback_kernel(const int* chosen, int* tokens, int* pos, int rows) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  if (r < rows) {
    tokens[r] = chosen[r];
    pos[r] += 1;
  }
}

// Inputs of a step from pinned host memory (tokens, positions and slots of `rows` rows, one after the other), and its result back into
// it.  The GPU reads and writes that memory itself: three copies by the copy engines and one back, each with a hand-over between
// engines, cost a decode step some 20 us more, torch's share of them included
// (one request of flash, three layers: 888 us a step with those, 870 so).  Neither kernel lets the next one start early, since those read the inputs before they
// wait (a graph's first kernel does not start early in any case).
__global__ void step_inputs_kernel(const int* host, int* tokens, int* pos, int* slot, int rows) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * rows) return;
  const int part = i / rows, r = i - part * rows;
  (part == 0 ? tokens : part == 1 ? pos : slot)[r] = __ldcv(host + i);
}
__global__ void step_result_kernel(const int* chosen, int* host, int rows) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < rows) host[r] = chosen[r];
}

}  // namespace ds41

using namespace ds41;

extern "C" int ds41_step_inputs(const int* host, int* tokens, int* pos, int* slot, int rows, void* stream) {
  if (host == nullptr || tokens == nullptr || pos == nullptr || slot == nullptr || rows <= 0 || rows > (1 << 28))
    return cudaErrorInvalidValue;
  step_inputs_kernel<<<(3 * rows + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(host, tokens, pos, slot, rows);
  return cudaGetLastError();
}

extern "C" int ds41_step_result(const int* chosen, int* host, int rows, void* stream) {
  if (chosen == nullptr || host == nullptr || rows <= 0) return cudaErrorInvalidValue;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  step_result_kernel<<<(rows + 255) / 256, 256, 0, st>>>(chosen, host, rows);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? e : cudaStreamSynchronize(st);
}

extern "C" int ds41_graph_step(void* graph_exec, const int* host_in, int* tokens, int* pos, int* slot, const int* chosen,
                               int* host_out, int rows, void* stream) {
  if (graph_exec == nullptr) return cudaErrorInvalidValue;
  int e = ds41_step_inputs(host_in, tokens, pos, slot, rows, stream);
  if (e != cudaSuccess) return e;
  e = cudaGraphLaunch(static_cast<cudaGraphExec_t>(graph_exec), static_cast<cudaStream_t>(stream));
  return e != cudaSuccess ? e : ds41_step_result(chosen, host_out, rows, stream);
}

extern "C" int ds41_decode_feedback(const int* chosen, int* tokens, int* pos, int rows, void* stream) {
  if (rows <= 0) return cudaErrorInvalidValue;
  return launch_pdl(decode_feedback_kernel, dim3((rows + 127) / 128), dim3(128), 0, static_cast<cudaStream_t>(stream),
                    chosen, tokens, pos, rows);
}

extern "C" int ds41_argmax_rows(const float* logits, long long ld, int rows, int vocab_local, int vocab_offset,
                                const uint32_t* mask, int mask_words, float* best_val, int* best_idx,
                                int* row_status, void* stream) {
  if (rows <= 0 || vocab_local <= 0) return cudaErrorInvalidValue;
  ArgmaxParams p{logits, ld, vocab_local, vocab_offset, mask, mask_words, best_val, best_idx, row_status};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (argmax_in_cluster(rows, vocab_local))
    return launch_pdl_cluster(argmax_rows_kernel<kArgmaxCtas, 512, 4>, dim3(rows * kArgmaxCtas), dim3(512), kArgmaxCtas, 0, st,
                              p);
  return launch_pdl(argmax_rows_kernel<1, 1024, 2>, dim3(rows), dim3(1024), 0, st, p);
}

extern "C" int ds41_argmax_merge(const float* const* vals, const int* const* idxs, int n_ranks, int rows, int* out,
                                 const uint32_t* const* wait_flags, const uint32_t* wait_epoch, int* status,
                                 void* stream) {
  if (n_ranks <= 0 || n_ranks > 8 || rows <= 0) return cudaErrorInvalidValue;
  MergeArgs p{};
  for (int k = 0; k < n_ranks; ++k) { p.vals[k] = vals[k]; p.idxs[k] = idxs[k]; }
  p.n_ranks = n_ranks; p.rows = rows; p.out = out;
  p.wait_flags = wait_flags; p.wait_epoch = wait_epoch; p.status = status;
  return launch_pdl(argmax_merge_kernel, dim3((rows + 127) / 128), dim3(128), 0, static_cast<cudaStream_t>(stream), p);
}

extern "C" int ds41_spec_accept(const int* inputs, const int* chosen, const int* first, const int* count, int reqs,
                                int max_emit, int eos, int* accepted, int* emit, int* n_emit, void* stream) {
  if (reqs <= 0 || max_emit <= 0) return cudaErrorInvalidValue;
  AcceptParams p{inputs, chosen, first, count, reqs, max_emit, eos, accepted, emit, n_emit};
  return launch_pdl(spec_accept_kernel, dim3((reqs + 63) / 64), dim3(64), 0, static_cast<cudaStream_t>(stream), p);
}
