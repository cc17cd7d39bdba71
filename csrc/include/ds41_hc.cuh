// What the hyper-connection kernels (hc.cu, hc_step.cu) share.
#pragma once
#include "ds41_ptx.cuh"

namespace ds41 {

// v / s in the manner of Markstein (Computation of elementary functions on the IBM RISC System/6000 processor, 1990): an
// approximate reciprocal, one Newton step, and the quotient corrected by its own remainder; for numbers whose reciprocals and
// quotients are normal or zero.  At most one unit of the last place off; the operator's own bits in all of 50 million pairs, of the
// mixes' range (divisors from 2^-20 to 8) and of far more.  Thirty-nine divisions in a row are what a row's mixes wait for, and
// this one is a chain of six instructions without a test (20 iterations of a 4 x 4 matrix 8060 cycles with the operator, 6250 so).
__device__ __forceinline__ float quotient(float v, float s) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
  r = fmaf(fmaf(-s, r, 1.0f), r, r);
  const float q = v * r;
  return fmaf(fmaf(-s, q, v), r, q);
}

// The 4 x 4 matrix that a warp's lanes 4 s + d hold (twice): softmax over d, then rows and columns divided by their sums in turn.
__device__ __forceinline__ float sinkhorn_4x4(float v, int iters, float eps) {
  auto over = [](float x, int o) {                  // the sum over d (o = 1) or s (o = 4)
    x += __shfl_xor_sync(0xffffffffu, x, o);
    return x + __shfl_xor_sync(0xffffffffu, x, 2 * o);
  };
  float mx = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
  v = __expf(v - mx);
  v = quotient(v, over(v, 1)) + eps;
  v = quotient(v, over(v, 4) + eps);
  for (int it = 1; it < iters; ++it) {
    v = quotient(v, over(v, 1) + eps);
    v = quotient(v, over(v, 4) + eps);
  }
  return v;
}

}  // namespace ds41
