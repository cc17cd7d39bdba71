// Grammar-mask token sampler on the GPU: one, two, four or eight 1024-thread CTAs per row.
//
// Same rule as the host oracle (csrc/core/sampler.cc): allow-mask -> temperature -> min_p -> top_k -> top_p ->
// categorical draw with a SplitMix64 (seed, position) uniform; greedy when T < 1e-5 or top_k == 1 (strict whole-row
// finiteness, lowest id wins ties).  Nothing is sorted.  The ranked order (scaled logit descending, id ascending) is
// handled with selections, digit by digit, over an order-preserving integer key:
//   * top-k   : select the k-th largest key by COUNT; ties at that key are admitted lowest id first
//   * top-p   : select by MASS the key at which the cumulative weight reaches top_p * total
//   * the draw: select by MASS the key at which the cumulative weight reaches u * nucleus mass, then the tie index
// Weights exp(scaled - max) are accumulated as 2^-40 fixed point in 64-bit integers, so every sum is independent of
// the order in which threads add and the result is bit-reproducible.  Without top_k / top_p the draw walks the
// survivors in token order (warps own consecutive tokens), as the oracle does.
// Parity target in the reference: native/cuda/kernels/v41_sampling_gpu.cu:238,523,921,1046,1701 (K1 prepare,
// K2 categorical, K3 top-k pivot, K4 membership / rank order, K5 nucleus) and v41_sampling_gpu.h:52-170.
#include <cooperative_groups.h>

#include <atomic>

#include "ds41_api.h"
#include "ds41_launch.cuh"

namespace cg = cooperative_groups;

namespace ds41 {

enum SampleStatus : int {
  kSampleOk = 0,
  kSampleEmpty = 1,
  kSampleNonFinite = 2,
  kSampleBadTemperature = 3,
  kSampleInternal = 5,
  kSampleBadParameter = 6,
};

constexpr int kSampleThreads = 1024;
constexpr double kFx = 1099511627776.0;   // 2^40

__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
__device__ __forceinline__ unsigned long long weight_fx(float scaled, float max_scaled) {
  return static_cast<unsigned long long>(exp(static_cast<double>(scaled - max_scaled)) * kFx + 0.5);
}
__device__ __forceinline__ bool mask_allows(const uint32_t* mask, int i) {
  return mask == nullptr || ((mask[i >> 5] >> (i & 31)) & 1u) != 0;
}
__device__ __forceinline__ float uniform01(unsigned long long seed, unsigned long long position) {
  const unsigned long long kDomain = 0x7f4a7c159e3779b9ull, kPhi = 0x9e3779b97f4a7c15ull;
  unsigned long long x = seed + kDomain + position * kPhi + kPhi;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  x ^= x >> 31;
  return static_cast<float>(static_cast<uint32_t>(x >> 40)) * (1.0f / 16777216.0f);
}

// A row is shared by a cluster of up to eight CTAs.  One CTA per row walked 517 KB up to fifteen times from L2 with a fraction of
// one SM's bandwidth: 780 us for sixteen rows of 129280 logits.  Now each CTA reads its part once, keeps the order keys of the
// scaled logits in shared memory, and only histograms, sums and short lists travel, through distributed shared memory.  Every CTA
// draws the same conclusions from the same integers, so there is no broadcast step and all control flow is uniform in the cluster.
// What is left is a chain of cluster barriers (2000 cycles each) and of passes over the keys (5000 to 7000 cycles); the reads from
// memory are 2 % of it.  So a selection sorts the row into 1024 bins of its own, of which the CTAs exchange 256 sums and then the
// four bins of one, and the draw looks at the nucleus' histogram again instead of making one: 16 rows with mixed filters 80 us
// with 256 bins and a histogram for every selection, 52 so; nucleus rows alone 109 and 72.
constexpr int kSampleMaxCluster = 8;
constexpr int kSampleMaxSlice = 49152;     // keys per CTA that fit its shared memory; longer slices are read again from L2
// A slice's first histogram has PER bins for each of the 256 that the CTAs exchange: four, or one beside the longest slices
constexpr int kSampleFineSlice = 45056;

struct SamplePart {                        // what one CTA found in its slice
  float best;
  int best_i;
  unsigned int allowed, bad;
};

constexpr int kSampleList = 512;           // candidates that are gathered and compared one by one instead of histogrammed
// Lists that solve_short() takes.  A shared search has three more barriers and a pass of one warp, 1.5 to 2 us: 16 rows of 129280 with a
// single filter of 40 tokens 45.1 us by it alone, 41.3 so; with nucleus as well 55.4 and 49.8.  Long lists are another matter: 64 rows of
// 4096, nucleus, 49 us without it, 33 so.  Lines from 48 to 192 measure the same.
constexpr int kSampleShort = 96;

struct SampleMember {
  uint32_t key, count;
  unsigned long long mass;                 // by count: the count
};

template <int PER>
struct SampleShared {
  static constexpr int kFineBins = 256 * PER;
  // A weight is counted in pieces of 14 bits, whose sums over a slice of up to 2^18 tokens fit 32 bits (64-bit additions in shared
  // memory are compare-and-swap loops: 22 us a pass); longer slices take the first words as 64-bit sums.
  // The first histogram of a selection, this slice's: 32nds (PER = 4) below the maximum, and the same added up to
  // eighths.
  unsigned int fine_cnt[kFineBins];
  alignas(8) unsigned int fine_mass[3][kFineBins];
  // histograms of the even and odd passes that follow: the other one may still be read by peers
  unsigned int cnt[2][256];
  alignas(8) unsigned int mass[2][3][256];
  unsigned int tot_cnt[256];
  unsigned long long tot_mass[256];
  SamplePart part[kSampleMaxCluster];
  unsigned long long slot[3][kSampleMaxCluster];      // one exchange each
  unsigned long long warp[kSampleThreads / 32];
  SamplePart warp_part[kSampleThreads / 32];
  unsigned long long total;                        // weight of a selection's candidates
  unsigned long long total_list;
  unsigned int low_key;
  double remaining;
  unsigned long long above_mass;
  unsigned int digit, tie_count, best_key, n_above;
  int token;
  unsigned int own_n, far_n[kSampleMaxCluster];
  uint2 own_list[kSampleList];                     // {key, token} of this CTA's members
  int n_list;                                      // members of the last selection that were gathered; -1: too many
  int list_id[kSampleList + 1];
  SampleMember list[kSampleList + 1];
};
constexpr int kSampleMostPieces = 1 << 18;         // 2^18 x 2^14 = 2^32

// This CTA's part of the row: tokens [id0, id0 + n), as order keys; 0 = the token is not allowed (no finite value has key 0).
struct SampleSlice {
  const uint32_t* keys;      // in shared memory, or null: made again from the logits
  const float* logits;
  const uint32_t* mask;
  int id0, n;
  float inv_t;
  bool wide;                 // weights are summed in 64 bits: some slice of the row is longer than kSampleMostPieces
  __device__ __forceinline__ uint32_t operator[](int i) const {
    if (keys != nullptr) return keys[i];
    return mask_allows(mask, id0 + i) ? order_key(__fmul_rn(logits[i], inv_t)) : 0u;
  }
};

// The candidate set of a selection: allowed tokens with key > excl, plus `tie_mult` tokens of key `tie_key`
// (the admitted part of a tie group cut by an earlier selection; tie_key <= excl whenever tie_mult > 0).
struct CandSet {
  uint32_t excl;
  uint32_t tie_key;
  unsigned long long tie_mult;
};

// The CTAs that share a row: a cluster, or one CTA by itself.
template <int CL>
struct SamplePeers {
  __device__ __forceinline__ unsigned rank() const { return CL == 1 ? 0u : cg::this_cluster().block_rank(); }
  __device__ __forceinline__ void sync() const {
    if constexpr (CL == 1) __syncthreads();
    else cg::this_cluster().sync();
  }
  template <class T>
  __device__ __forceinline__ T* of(T* mine, int rank) const {
    if constexpr (CL == 1) return mine;
    else return cg::this_cluster().map_shared_rank(mine, rank);
  }
};

// Sum over the cluster; `slot` is used once per launch, so no second barrier protects it.
template <int CL, int PER>
__device__ unsigned long long cluster_sum(SampleShared<PER>& sh, SamplePeers<CL> cl, int slot, unsigned long long v) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) sh.warp[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    unsigned long long mine = sh.warp[threadIdx.x];
    for (int off = 16; off > 0; off >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, off);
    if (threadIdx.x < CL) *cl.of(&sh.slot[slot][cl.rank()], threadIdx.x) = mine;
  }
  cl.sync();
  unsigned long long all = 0;
  for (int c = 0; c < CL; ++c) all += sh.slot[slot][c];
  return all;
}

// 32nds (PER = 4) below the maximum, highest first, the last bucket open: the first digit of a selection.  It spreads the tokens of
// a row over the bins, where the top byte of a key (sign and exponent) put a row into half a dozen: the lanes of a warp then met
// in the same counters and a pass took 40 us.
template <int PER>
__device__ __forceinline__ uint32_t bucket_of(uint32_t key, float max_scaled) {
  constexpr uint32_t kLast = 256u * PER - 1u;
  const float d = (max_scaled - key_value(key)) * (8.0f * PER);
  return kLast - (d >= static_cast<float>(kLast) ? kLast : static_cast<uint32_t>(d));
}

// Every CTA gathers the members of all slices that `is_member` names (fewer than kSampleList) and the tie group, if it takes
// part.
template <int CL, int PER, class F>
__device__ void gather_members(SampleShared<PER>& sh, SamplePeers<CL> cl, const SampleSlice& row, float max_scaled,
                               const CandSet& set, bool by_mass, bool tie, F is_member) {
  const int tid = threadIdx.x;
  for (int i = tid; i < row.n; i += kSampleThreads) {
    const uint32_t k = row[i];
    if (k > set.excl && is_member(k)) {
      const unsigned at = atomicAdd(&sh.own_n, 1u);
      if (at < kSampleList) sh.own_list[at] = make_uint2(k, static_cast<uint32_t>(row.id0 + i));
    }
  }
  cl.sync();
  if (tid < CL) sh.far_n[tid] = *cl.of(&sh.own_n, tid);
  __syncthreads();
  constexpr int kPer = kSampleThreads / CL;      // threads that read one peer's members
  const int from = min(tid / kPer, CL - 1);      // the last one's may be a few more
  int before = 0, n = 0;
#pragma unroll
  for (int r = 0; r < CL; ++r) {
    before = r == from ? n : before;
    n += static_cast<int>(sh.far_n[r]);
  }
  n = min(n, kSampleList);
  for (int i = tid - from * kPer; i < static_cast<int>(sh.far_n[from]) && before + i < kSampleList && tid < CL * kPer; i += kPer) {
    const uint2 m = *cl.of(&sh.own_list[i], from);
    sh.list[before + i] = {m.x, 1u, by_mass ? weight_fx(key_value(m.x), max_scaled) : 1ull};
    sh.list_id[before + i] = static_cast<int>(m.y);
  }
  if (tid == 0) {
    if (tie)
      sh.list[n] = {set.tie_key, static_cast<uint32_t>(set.tie_mult),
                    set.tie_mult * (by_mass ? weight_fx(key_value(set.tie_key), max_scaled) : 1ull)};
    sh.n_list = n;
  }
  __syncthreads();
}

// The highest key whose members and the ones above weigh at least the target (`frac` >= 0: that share of the list's weight).
// A short list: every thread sums what lies above its own member.
template <int PER>
__device__ uint32_t solve_short(SampleShared<PER>& sh, int total, double target, double frac) {
  const int tid = threadIdx.x;
  uint32_t key = 0, equal = 0, higher = 0, low = 0xFFFFFFFFu;
  unsigned long long above = 0, same = 0, all = 0;
  if (tid == 0) sh.best_key = 0;
  __syncthreads();
  if (tid < total) {
    key = sh.list[tid].key;
#pragma unroll 4
    for (int j = 0; j < total; ++j) {
      const SampleMember m = sh.list[j];
      all += m.mass;
      above += m.key > key ? m.mass : 0ull;
      same += m.key == key ? m.mass : 0ull;
      higher += m.key > key ? m.count : 0u;
      equal += m.key == key ? m.count : 0u;
      low = min(low, m.key);
    }
    if (frac >= 0.0) target = frac * static_cast<double>(all);
    // rounding can leave the target just above the total: then the lowest key present is the one
    if (static_cast<double>(above + same) >= target || key == low) atomicMax(&sh.best_key, key);
  }
  __syncthreads();
  const uint32_t best = sh.best_key;
  if (tid < total && key == best) {              // members of one key write the same
    sh.remaining = target - static_cast<double>(above);
    sh.tie_count = equal;
    sh.n_above = higher;
    if (frac >= 0.0) sh.total = all;
  }
  __syncthreads();
  return best;
}

// The same of any list: several lanes share a member and sum what is not below it, each over a part of the list.
template <int PER>
__device__ uint32_t solve_list(SampleShared<PER>& sh, bool tie, double target, double frac) {
  const int tid = threadIdx.x, total = sh.n_list + (tie ? 1 : 0);
  if (total <= kSampleShort) return solve_short(sh, total, target, frac);
  int per = 32;                                  // lanes per member
  while (per > 1 && total * per > kSampleThreads) per >>= 1;
  const int member = tid / per, part = tid % per;
  const bool live = member < total;
  const uint32_t key = live ? sh.list[member].key : 0u;
  unsigned long long upto = 0, all = 0;
  uint32_t low = 0xFFFFFFFFu;
  if (tid == 0) {
    sh.best_key = 0;
    sh.low_key = 0xFFFFFFFFu;
    sh.total_list = 0;
  }
  __syncthreads();
  if (live) {
#pragma unroll 4
    for (int j = part; j < total; j += per) {
      const SampleMember m = sh.list[j];
      upto += m.key >= key ? m.mass : 0ull;
    }
  }
  for (int o = per >> 1; o > 0; o >>= 1) upto += __shfl_xor_sync(0xffffffffu, upto, o);
  if (tid < total) {
    all = sh.list[tid].mass;
    low = sh.list[tid].key;
  }
  low = __reduce_min_sync(0xffffffffu, low);
  for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
  if ((tid & 31) == 0 && tid < total) {
    atomicMin(&sh.low_key, low);
    atomicAdd(&sh.total_list, all);
  }
  __syncthreads();
  all = sh.total_list;
  if (frac >= 0.0) target = frac * static_cast<double>(all);
  // rounding can leave the target just above the total: then the lowest key present is the one
  if (live && (static_cast<double>(upto) >= target || key == sh.low_key)) atomicMax(&sh.best_key, key);
  __syncthreads();
  const uint32_t best = sh.best_key;
  if (tid < 32) {                                // what lies above it
    unsigned long long above = 0;
    uint32_t equal = 0, higher = 0;
    for (int j = tid; j < total; j += 32) {
      const SampleMember m = sh.list[j];
      above += m.key > best ? m.mass : 0ull;
      equal += m.key == best ? m.count : 0u;
      higher += m.key > best ? m.count : 0u;
    }
    equal = __reduce_add_sync(0xffffffffu, equal);
    higher = __reduce_add_sync(0xffffffffu, higher);
    for (int o = 16; o > 0; o >>= 1) above += __shfl_xor_sync(0xffffffffu, above, o);
    if (tid == 0) {
      sh.remaining = target - static_cast<double>(above);
      sh.tie_count = equal;
      sh.n_above = higher;
      if (frac >= 0.0) sh.total = all;
    }
  }
  __syncthreads();
  return best;
}

// Selection by five digits (the bucket, then the bytes of the key), high keys first.  by_mass: find the key at which the running
// weight reaches the target; else the key at which the running count reaches it.  `frac` >= 0: the target is that share of the
// set's weight, which is left in sh.total.
// `narrowed`: the set is what the selection before this one, by weight too, left of its own: whole bins above the bin of
// set.excl, whose histogram stands, and a part of that bin; one look at the histogram then takes the place of a pass.
// On return sh.remaining is what the ties at the returned key must still supply and sh.tie_count how many candidates carry it.
// `pass` counts the histograms of the launch.
template <int CL, int PER>
__device__ uint32_t radix_select(SampleShared<PER>& sh, SamplePeers<CL> cl, const SampleSlice& row, float max_scaled, CandSet set,
                                 bool by_mass, double target, double frac, bool narrowed, int& pass) {
  const int tid = threadIdx.x, lane = tid & 31;
  constexpr int kFineBins = 256 * PER;
  auto add_mass = [&](unsigned int* mass, int bins, uint32_t d, unsigned long long w) {
    if (row.wide) {
      atomicAdd(reinterpret_cast<unsigned long long*>(mass) + d, w);
      return;
    }
    constexpr unsigned kPiece = (1u << 14) - 1;
    const unsigned a = static_cast<unsigned>(w) & kPiece, b = static_cast<unsigned>(w >> 14) & kPiece;
    const unsigned c = static_cast<unsigned>(w >> 28);
    if (a != 0) atomicAdd(mass + d, a);
    if (b != 0) atomicAdd(mass + bins + d, b);
    if (c != 0) atomicAdd(mass + 2 * bins + d, c);
  };
  auto whole = [&](const unsigned int* mass, int bins, uint32_t d) -> unsigned long long {
    if (row.wide) return reinterpret_cast<const unsigned long long*>(mass)[d];
    return mass[d] + (static_cast<unsigned long long>(mass[bins + d]) << 14) +
           (static_cast<unsigned long long>(mass[2 * bins + d]) << 28);
  };
  const uint32_t floor_bin = narrowed ? bucket_of<PER>(set.excl, max_scaled) : 0u;
  // Warp 0: the first of the 256 bins, from the highest down, whose running weight reaches the target.
  auto scan = [&](bool first) {
    // eight bins per lane from the highest down: the first bin in use whose running sum reaches the target
    unsigned long long sum = 0;
    unsigned members = 0;
    auto bin_of = [&](int j) { return 255 - 8 * lane - j; };
    auto out = [&](int d) { return first && d < static_cast<int>(floor_bin / PER); };
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (out(bin_of(j))) continue;
      sum += sh.tot_mass[bin_of(j)];
      members += sh.tot_cnt[bin_of(j)];
    }
    const bool used = members != 0;
    unsigned long long incl = sum;
    unsigned higher = members;
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, off);
      const unsigned more = __shfl_up_sync(0xffffffffu, higher, off);
      if (lane >= off) {
        incl += up;
        higher += more;
      }
    }
    higher -= members;
    const unsigned long long all = __shfl_sync(0xffffffffu, incl, 31);
    if (first && frac >= 0.0) target = frac * static_cast<double>(all);
    const unsigned reach = __ballot_sync(0xffffffffu, used && static_cast<double>(incl) >= target);
    const unsigned any = __ballot_sync(0xffffffffu, used);
    // rounding can leave the target just above the total: then the selection ends on the lowest key present
    const int owner = reach != 0 ? __ffs(reach) - 1 : (any != 0 ? 31 - __clz(any) : 0);
    if (lane == owner) {
      unsigned long long acc = incl - sum, at = acc;
      int pick = -1;
      for (int j = 0; j < 8; ++j) {
        const int d = bin_of(j);
        if (out(d) || sh.tot_cnt[d] == 0) continue;
        if (pick >= 0) higher += sh.tot_cnt[pick];
        pick = d;
        at = acc;
        acc += sh.tot_mass[d];
        if (reach != 0 && static_cast<double>(acc) >= target) break;
      }
      if (pick < 0) pick = 0;
      sh.digit = static_cast<unsigned int>(pick);
      sh.above_mass = at;
      sh.tie_count = sh.tot_cnt[pick];
      sh.n_above = first ? higher : sh.n_above + higher;
      if (first) sh.total = all;
    }
    __syncwarp();
    if (!first) {
      if (lane == 0) sh.remaining = target - static_cast<double>(sh.above_mass);
      return;
    }
    // the bin that the four bins of its eighth hide: lane (peer, bin) reads, all lanes add
    const uint32_t coarse = sh.digit;
    const int sub = lane & (PER - 1);
    const uint32_t d = coarse * PER + sub;
    unsigned c = 0;
    unsigned long long m = 0;
    for (int r = lane / PER; r < CL; r += 32 / PER) {
      c += *cl.of(&sh.fine_cnt[d], r);
      if (by_mass) m += whole(cl.of(sh.fine_mass[0], r), kFineBins, d);
    }
#pragma unroll
    for (int o = PER; o < 32; o <<= 1) {
      c += __shfl_xor_sync(0xffffffffu, c, o);
      m += __shfl_xor_sync(0xffffffffu, m, o);
    }
    // (narrowed: the lowest bin counts more than the set has of it, and nothing below it is looked at)
    if (set.tie_mult > 0 && bucket_of<PER>(set.tie_key, max_scaled) == d) {
      c += static_cast<unsigned>(set.tie_mult);
      m += set.tie_mult * weight_fx(key_value(set.tie_key), max_scaled);
    }
    if (!by_mass) m = c;
    unsigned long long acc = sh.above_mass, at = acc;
    unsigned above = sh.n_above, before = above, count = 0;
    int pick = -1;
#pragma unroll
    for (int k = PER - 1; k >= 0; --k) {
      const unsigned ck = __shfl_sync(0xffffffffu, c, k);
      const unsigned long long mk = __shfl_sync(0xffffffffu, m, k);
      const bool done = pick >= 0 && reach != 0 && static_cast<double>(acc) >= target;
      if (!done && ck != 0 && coarse * PER + k >= floor_bin) {
        pick = k;
        at = acc;
        before = above;
        count = ck;
        acc += mk;
        above += ck;
      }
    }
    if (lane == 0) {
      if (pick < 0) pick = 0;
      sh.remaining = target - static_cast<double>(at);
      sh.digit = coarse * PER + pick;
      sh.tie_count = count;
      sh.n_above = before;
    }
  };
  // ---- the first digit
  if (!narrowed) {
    for (int i = tid; i < kFineBins; i += kSampleThreads)
      sh.fine_cnt[i] = sh.fine_mass[0][i] = sh.fine_mass[1][i] = sh.fine_mass[2][i] = 0;
    __syncthreads();
    // Integer sums: the result does not depend on the order or the grouping of the additions.
    for (int base = 0; base < row.n; base += kSampleThreads) {
      const uint32_t k = base + tid < row.n ? row[base + tid] : 0u;
      if (k <= set.excl) continue;
      const uint32_t d = bucket_of<PER>(k, max_scaled);
      atomicAdd(&sh.fine_cnt[d], 1u);
      if (by_mass) add_mass(sh.fine_mass[0], kFineBins, d, weight_fx(key_value(k), max_scaled));
    }
    __syncthreads();
    unsigned int* cnt = sh.cnt[pass & 1];
    unsigned long long* mass = reinterpret_cast<unsigned long long*>(sh.mass[pass & 1][0]);
    ++pass;
    if (tid < 256) {
      unsigned c = 0;
      unsigned long long m = 0;
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        c += sh.fine_cnt[tid * PER + k];
        if (by_mass) m += whole(sh.fine_mass[0], kFineBins, tid * PER + k);
      }
      cnt[tid] = c;
      mass[tid] = m;
    }
    cl.sync();
    if (tid < 256) {
      unsigned int c = 0;
      unsigned long long m = 0;
#pragma unroll
      for (int r = 0; r < CL; ++r) {
        c += *cl.of(&cnt[tid], r);
        if (by_mass) m += *cl.of(&mass[tid], r);
      }
      if (set.tie_mult > 0 && bucket_of<PER>(set.tie_key, max_scaled) / PER == static_cast<uint32_t>(tid)) {
        c += static_cast<unsigned int>(set.tie_mult);
        if (by_mass) m += set.tie_mult * weight_fx(key_value(set.tie_key), max_scaled);
      }
      sh.tot_cnt[tid] = c;
      sh.tot_mass[tid] = by_mass ? m : c;
    }
  } else {
    cl.sync();                                   // peers are done with this CTA's former members
  }
  if (tid == 0) {
    sh.own_n = 0;
    sh.n_list = -1;
  }
  __syncthreads();
  if (tid < 32) scan(true);
  __syncthreads();
  target = sh.remaining;
  const uint32_t bucket = sh.digit;
  if (sh.tie_count < kSampleList) {
    const bool tie = set.tie_mult > 0 && bucket_of<PER>(set.tie_key, max_scaled) == bucket;
    const unsigned above = sh.n_above;
    gather_members(sh, cl, row, max_scaled, set, by_mass, tie,
                   [&](uint32_t k) { return bucket_of<PER>(k, max_scaled) == bucket; });
    const uint32_t key = solve_list(sh, tie, target, -1.0);
    if (tid == 0) sh.n_above += above;
    __syncthreads();
    return key;
  }
  // ---- too many tokens in one bin: the bytes of their keys
  uint32_t prefix = 0, prefix_mask = 0;
  for (int shift = 24; shift >= 0; shift -= 8, ++pass) {
    unsigned int* cnt = sh.cnt[pass & 1];
    unsigned int(*mass)[256] = sh.mass[pass & 1];
    if (tid < 256) cnt[tid] = mass[0][tid] = mass[1][tid] = mass[2][tid] = 0;
    __syncthreads();
    auto member = [&](uint32_t k) { return bucket_of<PER>(k, max_scaled) == bucket && (k & prefix_mask) == prefix; };
    auto digit = [&](uint32_t k) { return (k >> shift) & 255u; };
    // Lanes of a warp that hit the same digit add once, since the tokens that are left share their top bytes.
    for (int base = 0; base < row.n; base += kSampleThreads) {
      const uint32_t k = base + tid < row.n ? row[base + tid] : 0u;
      const bool act = k > set.excl && member(k);
      if (!__any_sync(0xffffffffu, act)) continue;
      const uint32_t d = digit(k);
      const unsigned peers = __match_any_sync(0xffffffffu, act ? d : 256u);
      if (act) {
        if (by_mass) add_mass(mass[0], 256, d, weight_fx(key_value(k), max_scaled));
        if (lane == __ffs(peers) - 1) atomicAdd(&cnt[d], static_cast<unsigned>(__popc(peers)));
      }
    }
    if (cl.rank() == 0 && tid == 0 && set.tie_mult > 0 && member(set.tie_key))
      atomicAdd(&cnt[digit(set.tie_key)], static_cast<unsigned int>(set.tie_mult));
    cl.sync();
    if (tid < 256) {
      unsigned int c = 0;
      unsigned long long m = 0;
#pragma unroll
      for (int r = 0; r < CL; ++r) {
        c += *cl.of(&cnt[tid], r);
        if (by_mass) m += whole(cl.of(mass[0], r), 256, tid);
      }
      if (by_mass && set.tie_mult > 0 && member(set.tie_key) && digit(set.tie_key) == static_cast<uint32_t>(tid))
        m += set.tie_mult * weight_fx(key_value(set.tie_key), max_scaled);
      sh.tot_cnt[tid] = c;
      sh.tot_mass[tid] = by_mass ? m : c;
    }
    __syncthreads();
    if (tid < 32) scan(false);
    __syncthreads();
    target = sh.remaining;
    prefix |= sh.digit << shift;
    prefix_mask |= 255u << shift;
  }
  return prefix;
}

template <int CL, int PER>
__global__ void __launch_bounds__(kSampleThreads)
sample_rows_kernel(const float* __restrict__ logits, long long ld, int vocab, const uint32_t* __restrict__ masks,
                   int mask_words, const ds41_sample_row* __restrict__ rows, int* __restrict__ tokens,
                   int* __restrict__ status) {
  __shared__ SampleShared<PER> sh;
  extern __shared__ uint32_t key_store[];
  pdl_launch_dependents();
  pdl_wait();
  const SamplePeers<CL> cl;
  const int rank = static_cast<int>(cl.rank()), row = blockIdx.x / CL;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const ds41_sample_row p = rows[row];
  const uint32_t* mask = (masks != nullptr && p.mask_row >= 0) ? masks + 1ll * p.mask_row * mask_words : nullptr;
  // every return below is taken by the whole cluster at once, and after the last look into a peer's memory
  auto finish = [&](int st, int tok) {
    cl.sync();
    if (rank == 0 && tid == 0) {
      status[row] = st;
      if (st == kSampleOk) tokens[row] = tok;
    }
  };
  if (!(p.temperature >= 0.0f) || isinf(p.temperature)) return finish(kSampleBadTemperature, 0);
  if (!(p.top_p > 0.0f) || !(p.min_p >= 0.0f) || p.min_p > 1.0f) return finish(kSampleBadParameter, 0);
  // a peer's shared memory may be touched once all CTAs of the cluster run: the wait hides behind the slice's loads
  if constexpr (CL > 1) cg::cluster_group::barrier_arrive();
  const bool greedy = p.temperature < 1e-5f || p.top_k == 1;
  const float inv_t = greedy ? 1.0f : 1.0f / p.temperature;

  // ---- the slice: order keys, finiteness, allowed count, maximum (greedy: arg max with the lowest id on ties)
  const int slice = ((vocab + CL - 1) / CL + 31) & ~31;
  SampleSlice own;
  own.id0 = min(vocab, rank * slice);
  own.n = min(vocab, own.id0 + slice) - own.id0;
  own.logits = logits + 1ll * row * ld + own.id0;
  own.mask = mask;
  own.inv_t = inv_t;
  own.keys = slice <= kSampleMaxSlice && (CL > 1 || !greedy) ? key_store : nullptr;
  own.wide = slice > kSampleMostPieces;
  SamplePart mine{-INFINITY, -1, 0u, 0u};
  auto take = [&](int i, float v) {
    const bool ok = mask_allows(mask, own.id0 + i);
    if (greedy ? !isfinite(v) : ok && (isnan(v) || v == INFINITY)) mine.bad = 1u;
    const float s = __fmul_rn(v, inv_t);
    if (ok) {
      ++mine.allowed;
      if (mine.best_i < 0 || s > mine.best) { mine.best = s; mine.best_i = own.id0 + i; }    // ascending: first maximum kept
    }
    if (own.keys != nullptr) key_store[i] = ok ? order_key(s) : 0u;
  };
  int done = 0;
  if ((reinterpret_cast<uintptr_t>(own.logits) & 15) == 0) {
    const int n4 = own.n >> 2;
    const float4* src = reinterpret_cast<const float4*>(own.logits);
    for (int base = 0; base < n4; base += 4 * kSampleThreads) {
      float4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int q = base + j * kSampleThreads + tid;
        if (q < n4) v[j] = src[q];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int q = base + j * kSampleThreads + tid;
        if (q < n4) {
          take(4 * q, v[j].x);
          take(4 * q + 1, v[j].y);
          take(4 * q + 2, v[j].z);
          take(4 * q + 3, v[j].w);
        }
      }
    }
    done = 4 * n4;
  }
  for (int i = done + tid; i < own.n; i += kSampleThreads) take(i, own.logits[i]);
  auto merge = [](SamplePart& a, const SamplePart& b) {
    a.allowed += b.allowed;
    a.bad |= b.bad;
    if (b.best_i >= 0 && (a.best_i < 0 || b.best > a.best || (b.best == a.best && b.best_i < a.best_i))) {
      a.best = b.best;
      a.best_i = b.best_i;
    }
  };
  auto merge_warp = [&](SamplePart& a) {
    for (int off = 16; off > 0; off >>= 1) {
      SamplePart o;
      o.best = __shfl_xor_sync(0xffffffffu, a.best, off);
      o.best_i = __shfl_xor_sync(0xffffffffu, a.best_i, off);
      o.allowed = __shfl_xor_sync(0xffffffffu, a.allowed, off);
      o.bad = __shfl_xor_sync(0xffffffffu, a.bad, off);
      merge(a, o);
    }
  };
  static_assert(kSampleThreads == 1024, "one warp merges the warps");
  merge_warp(mine);
  if (lane == 0) sh.warp_part[warp] = mine;
  __syncthreads();
  if constexpr (CL > 1) cg::cluster_group::barrier_wait();
  if (warp == 0) {
    mine = sh.warp_part[lane];
    merge_warp(mine);
    if (lane < CL) *cl.of(&sh.part[rank], lane) = mine;
  }
  cl.sync();
  SamplePart all = sh.part[0];
  for (int c = 1; c < CL; ++c) merge(all, sh.part[c]);
  if (all.bad != 0u) return finish(kSampleNonFinite, 0);
  if (all.best_i < 0 || all.allowed == 0) return finish(kSampleEmpty, 0);
  if (greedy) return finish(kSampleOk, all.best_i);
  const float max_scaled = all.best;
  if (!isfinite(max_scaled)) return finish(kSampleEmpty, 0);

  const float u = fminf(fmaxf(uniform01(p.seed, p.position), 0.0f), 0.99999994f);
  const float min_scaled = p.min_p > 0.0f ? max_scaled + logf(p.min_p) : -INFINITY;
  // survivors: key >= key(min_scaled)  <=>  key > excl
  const uint32_t excl0 = p.min_p > 0.0f ? order_key(min_scaled) - 1u : 0u;
  const bool filtered = p.top_k > 0 || p.top_p < 1.0f;

  if (CL == 1 && !filtered) {
    // ---- categorical over the survivors in token order: every thread owns consecutive tokens, an odd number of them, so that
    // the threads of a warp read different banks
    const int seg = ((own.n + kSampleThreads - 1) / kSampleThreads) | 1;
    const int i0 = min(own.n, tid * seg), i1 = min(own.n, i0 + seg);
    auto weight = [&](int i) -> unsigned long long {
      const uint32_t k = own[i];
      return k > excl0 ? weight_fx(key_value(k), max_scaled) : 0ull;
    };
    unsigned long long sum = 0;
    for (int i = i0; i < i1; ++i) sum += weight(i);
    unsigned long long before = sum;
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned long long up = __shfl_up_sync(0xffffffffu, before, off);
      if (lane >= off) before += up;
    }
    before -= sum;
    const unsigned long long total = cluster_sum(sh, cl, 0, sum);
    for (int w = 0; w < warp; ++w) before += sh.warp[w];
    const double target = static_cast<double>(u) * static_cast<double>(total);
    if (tid == 0) sh.token = -1;
    __syncthreads();
    // the first thread whose running sum reaches the target owns the draw
    if (sum > 0 && static_cast<double>(before + sum) >= target && (static_cast<double>(before) < target || before == 0)) {
      for (int i = i0; i < i1; ++i) {
        before += weight(i);
        if (before > 0 && static_cast<double>(before) >= target) {
          sh.token = i;
          break;
        }
      }
    }
    __syncthreads();
    if (sh.token < 0) {                              // rounding left the target above every sum: the last survivor wins
      int last = -1;
      for (int i = i1 - 1; i >= i0 && last < 0; --i)
        if (own[i] > excl0) last = i;
      if (last >= 0) atomicMax(&sh.token, last);
      __syncthreads();
    }
    return finish(sh.token >= 0 ? kSampleOk : kSampleEmpty, sh.token);
  }
  if (!filtered) {
    // ---- categorical over the survivors in token order: a warp owns consecutive tokens, 32 at a time
    const int per_warp = ((own.n + kSampleThreads / 32 - 1) / (kSampleThreads / 32) + 31) & ~31;
    const int w0 = min(own.n, warp * per_warp), w1 = min(own.n, w0 + per_warp);
    auto weight = [&](int i) -> unsigned long long {
      const uint32_t k = i < w1 ? own[i] : 0u;
      return k > excl0 ? weight_fx(key_value(k), max_scaled) : 0ull;
    };
    unsigned long long sum = 0;
    for (int i = w0 + lane; i < w1; i += 32) sum += weight(i);
    const unsigned long long total = cluster_sum(sh, cl, 0, sum);
    const double target = static_cast<double>(u) * static_cast<double>(total);
    unsigned long long before = 0;
    for (int c = 0; c < rank; ++c) before += sh.slot[0][c];
    for (int w = 0; w < warp; ++w) before += sh.warp[w];
    const unsigned long long in_warp = sh.warp[warp];
    if (tid == 0) sh.token = -1;
    __syncthreads();
    // the first warp whose running sum reaches the target owns the draw
    if (in_warp > 0 && static_cast<double>(before + in_warp) >= target && (static_cast<double>(before) < target || before == 0)) {
      for (int i0 = w0; i0 < w1; i0 += 32) {
        unsigned long long incl = weight(i0 + lane);
        for (int off = 1; off < 32; off <<= 1) {
          const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, off);
          if (lane >= off) incl += up;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, before + incl > 0 && static_cast<double>(before + incl) >= target);
        if (hit != 0) {
          if (lane == 0) sh.token = own.id0 + i0 + __ffs(hit) - 1;
          break;
        }
        before += __shfl_sync(0xffffffffu, incl, 31);
      }
    }
    __syncthreads();
    // at most one CTA drew; where rounding left the target above every sum, the last survivor wins
    int last = sh.token;
    const int drawn = static_cast<int>(cluster_sum(sh, cl, 1, tid == 0 && last >= 0 ? 1ull + last : 0ull)) - 1;
    if (drawn >= 0) return finish(kSampleOk, drawn);
    last = -1;
    for (int i = tid; i < own.n; i += kSampleThreads)
      if (own[i] > excl0) last = max(last, i);
    last = __reduce_max_sync(0xffffffffu, last);
    if (lane == 0) atomicMax(&sh.token, last);
    __syncthreads();
    if (tid < CL)
      *cl.of(&sh.slot[2][rank], tid) = sh.token >= 0 ? 1ull + own.id0 + sh.token : 0ull;
    cl.sync();
    unsigned long long top = 0;
    for (int c = 0; c < CL; ++c) top = max(top, sh.slot[2][c]);
    return finish(top > 0 ? kSampleOk : kSampleEmpty, static_cast<int>(top) - 1);
  }

  // ---- ranked path
  CandSet set{excl0, 0u, 0ull};
  int pass = 0;
  // Once few candidates are left they are gathered, and what is still to be selected among them takes no more passes.
  bool gathered = false;
  auto gather_all = [&]() {
    const unsigned left = sh.n_above;              // candidates above the key just selected, without the tie group
    __syncthreads();
    if (left >= kSampleList) return;
    cl.sync();                                     // peers are done with this CTA's former members
    if (tid == 0) sh.own_n = 0;
    __syncthreads();
    gather_members(sh, cl, own, max_scaled, set, true, true, [](uint32_t) { return true; });
    gathered = true;
  };
  bool narrowed = false;                           // the last selection's histogram holds the set's bins
  auto select = [&](double target, double frac) {
    return gathered ? solve_list(sh, true, target, frac)
                    : radix_select(sh, cl, own, max_scaled, set, true, target, frac, narrowed, pass);
  };
  unsigned long long survivors = all.allowed;
  if (p.min_p > 0.0f) {
    unsigned long long n = 0;
    for (int i = tid; i < own.n; i += kSampleThreads) n += own[i] > excl0 ? 1 : 0;
    survivors = cluster_sum(sh, cl, 0, n);
  }
  if (survivors == 0) return finish(kSampleEmpty, 0);
  if (p.top_k > 0 && static_cast<unsigned long long>(p.top_k) < survivors) {
    const uint32_t pk = radix_select(sh, cl, own, max_scaled, set, false, static_cast<double>(p.top_k), -1.0, false,
                                     pass);
    set.excl = pk;
    set.tie_key = pk;
    set.tie_mult = static_cast<unsigned long long>(fmin(fmax(sh.remaining, 1.0), static_cast<double>(sh.tie_count)));
    gather_all();
  }
  double draw_of = -1.0, draw_frac = static_cast<double>(u);
  if (p.top_p < 1.0f) {
    const uint32_t pp = select(0.0, static_cast<double>(p.top_p));
    // tot_* keep the first histogram unless the selection went on to the bytes of the keys, or had a list to begin with
    narrowed = !gathered && sh.n_list >= 0;
    const double target = static_cast<double>(p.top_p) * static_cast<double>(sh.total);
    const double need = sh.remaining;
    const unsigned long long ties = sh.tie_count;
    const double w = static_cast<double>(weight_fx(key_value(pp), max_scaled));
    unsigned long long take = w > 0.0 ? static_cast<unsigned long long>(ceil(need / w)) : ties;
    if (take < 1) take = 1;
    if (take > ties) take = ties;
    draw_of = static_cast<double>(u) * ((target - need) + static_cast<double>(take) * w);
    draw_frac = -1.0;
    set.excl = pp;
    set.tie_key = pp;
    set.tie_mult = take;
    gather_all();
  }
  // ---- the draw
  const uint32_t dk = select(draw_of, draw_frac);
  const double need = sh.remaining;
  const unsigned long long ties = sh.tie_count;
  const double w = static_cast<double>(weight_fx(key_value(dk), max_scaled));
  long long tie_index = w > 0.0 ? static_cast<long long>(ceil(need / w)) - 1 : 0;
  if (tie_index < 0) tie_index = 0;
  if (tie_index > static_cast<long long>(ties) - 1) tie_index = static_cast<long long>(ties) - 1;
  if (sh.n_list >= 0 && !(set.tie_mult > 0 && dk == set.tie_key)) {
    // every token of that key is in the list: the one with exactly tie_index smaller ids among them
    if (tid < sh.n_list && sh.list[tid].key == dk) {
      int before = 0;
      for (int j = 0; j < sh.n_list; ++j) before += sh.list[j].key == dk && sh.list_id[j] < sh.list_id[tid] ? 1 : 0;
      if (before == tie_index && rank == 0) {
        status[row] = kSampleOk;
        tokens[row] = sh.list_id[tid];
      }
    }
    cl.sync();                                     // peers may still gather from this CTA
    return;
  }
  // the tie_index-th allowed token with key == dk in id order: the CTA that holds it, then its first warp, 32 tokens at a time
  unsigned long long eq = 0;
  for (int i = tid; i < own.n; i += kSampleThreads) eq += own[i] == dk ? 1 : 0;
  cluster_sum(sh, cl, 1, eq);
  long long before = 0;
  int holder = -1;
  for (int c = 0; c < CL; ++c) {
    const long long here = static_cast<long long>(sh.slot[1][c]);
    if (holder < 0 && tie_index < before + here) holder = c;
    if (holder < 0) before += here;
  }
  if (holder < 0) return finish(kSampleInternal, 0);
  if (rank == holder && warp == 0) {
    int rest = static_cast<int>(tie_index - before);
    for (int i0 = 0; i0 < own.n; i0 += 32) {
      unsigned hit = __ballot_sync(0xffffffffu, i0 + lane < own.n && own[i0 + lane] == dk);
      const int n = __popc(hit);
      if (rest >= n) {
        rest -= n;
        continue;
      }
      for (; rest > 0; --rest) hit &= hit - 1;
      if (lane == 0) {
        status[row] = kSampleOk;
        tokens[row] = own.id0 + i0 + __ffs(hit) - 1;
      }
      break;
    }
  }
  cl.sync();
}

}  // namespace ds41

using namespace ds41;

template <int CL, int PER>
static int launch_sample_as(const float* logits, long long ld, int rows, int vocab, const uint32_t* masks, int mask_words,
                            const ds41_sample_row* params, int* tokens, int* status, cudaStream_t stream) {
  const int slice = ((vocab + CL - 1) / CL + 31) & ~31;
  const size_t smem = slice <= kSampleMaxSlice ? 4ull * slice : 0;
  constexpr int kMost = PER > 1 ? kSampleFineSlice : kSampleMaxSlice;
  static std::atomic<bool> configured[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev].load(std::memory_order_acquire)) {
    const cudaError_t e = cudaFuncSetAttribute(sample_rows_kernel<CL, PER>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kMost);
    if (e != cudaSuccess) return e;
    configured[dev].store(true, std::memory_order_release);
  }
  if constexpr (CL == 1)
    return launch_pdl(sample_rows_kernel<CL, PER>, dim3(rows), dim3(kSampleThreads), smem, stream, logits, ld, vocab, masks,
                      mask_words, params, tokens, status);
  else
    return launch_pdl_cluster(sample_rows_kernel<CL, PER>, dim3(rows * CL), dim3(kSampleThreads), CL, smem, stream, logits, ld,
                              vocab, masks, mask_words, params, tokens, status);
}

template <int CL>
static int launch_sample(const float* logits, long long ld, int rows, int vocab, const uint32_t* masks, int mask_words,
                         const ds41_sample_row* params, int* tokens, int* status, cudaStream_t stream) {
  const int slice = ((vocab + CL - 1) / CL + 31) & ~31;
  return slice > kSampleFineSlice && slice <= kSampleMaxSlice
             ? launch_sample_as<CL, 1>(logits, ld, rows, vocab, masks, mask_words, params, tokens, status, stream)
             : launch_sample_as<CL, 4>(logits, ld, rows, vocab, masks, mask_words, params, tokens, status, stream);
}

// CTAs that share a row.  A row alone is fastest over eight; but about 15 clusters of eight run at once, 36 of four, 74 of two
// and 148 single CTAs, and every CTA more costs its barriers, which short rows do not earn back.  Slices should stay in shared
// memory.  What the rows ask for is known on the device alone, so the line is drawn by mixed passes; greedy rows by themselves,
// which have a kernel of their own (argmax_rows), and min-p rows lose by it where many rows are long (64 x 129280: 17 -> 32 and
// 57 -> 64 us).  us for rows that ask for plain temperature, nucleus, top-k and min-p in turn, over 8 / 4 / 2 / 1 CTAs (and one
// CTA that reads its row from L2 up to fifteen times):
//   2000 columns    8 rows  17 /  16 /  16 /   13  (67)     64 rows   61 /  35 /  30 /   27  (72)
//   16000 columns                                           64 rows   84 /  52 /  38 /   41 (152)
//   30000 columns  16 rows  34 /  38 /  47 /   64 (244)     64 rows   83 /  60 /  62 /   78 (253)
//                                                          148 rows  196 / 119 /  88 /   72 (250)
//   65536 columns  20 rows  51 /  61 /  99 /  213 (476)     64 rows  105 /  94 / 189 /  407 (480)
//   129280 columns 16 rows  68 / 100 / 235 /  419 (761)     64 rows  144 / 197 / 766 / 1508 (853)
//                                                          100 rows  222 / 178 / 393 / 1141 (855)
static int sample_ctas(int rows, int vocab) {
  if (vocab <= 4096) return 1;
  if (vocab <= kSampleMaxSlice) {
    if (vocab > 16384 && rows <= (vocab <= 32768 ? 15 : 24)) return 8;
    return rows <= 36 ? 4 : rows <= 74 ? 2 : 1;
  }
  if (vocab <= 2 * kSampleMaxSlice) return rows <= 40 ? 8 : rows <= 100 ? 4 : 2;
  return rows <= 64 || vocab > 4 * kSampleMaxSlice ? 8 : 4;
}

extern "C" int ds41_sample_rows(const float* logits, long long ld, int rows, int vocab, const uint32_t* masks,
                                int mask_words, const ds41_sample_row* params, int* tokens, int* status, void* stream) {
  if (logits == nullptr || params == nullptr || tokens == nullptr || status == nullptr || rows <= 0 || vocab <= 0)
    return cudaErrorInvalidValue;
  if (masks != nullptr && mask_words != (vocab + 31) / 32) return cudaErrorInvalidValue;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (sample_ctas(rows, vocab)) {
    case 8: return launch_sample<8>(logits, ld, rows, vocab, masks, mask_words, params, tokens, status, st);
    case 4: return launch_sample<4>(logits, ld, rows, vocab, masks, mask_words, params, tokens, status, st);
    case 2: return launch_sample<2>(logits, ld, rows, vocab, masks, mask_words, params, tokens, status, st);
    default: return launch_sample<1>(logits, ld, rows, vocab, masks, mask_words, params, tokens, status, st);
  }
}
