// Deterministic compensated FP64 reductions shared by the diagnostics and
// the adjoint: compensated (sum, error) pairs per thread, fixed-order block
// trees.
#pragma once
#include <cuda_runtime.h>

namespace bgk {

struct KS { double s, c; };
// Compensated step: the exact rounding error of a.s + v (Knuth's TwoSum, no
// comparison of the magnitudes) goes into a.c. Explicit _rn operations keep it
// free of FMA contraction.
__device__ __forceinline__ void kadd(KS& a, double v) {
  const double t = __dadd_rn(a.s, v);
  const double z = __dsub_rn(t, a.s);
  a.c = __dadd_rn(a.c, __dadd_rn(__dsub_rn(a.s, __dsub_rn(t, z)), __dsub_rn(v, z)));
  a.s = t;
}
__device__ __forceinline__ void kcomb(KS& a, const KS& b) {
  kadd(a, b.s);
  a.c = __dadd_rn(a.c, b.c);
}

// Fixed-order block reduction of one quantity; thread 0 returns the result.
__device__ __forceinline__ KS block_reduce(KS v, KS* sh) {
  const int t = threadIdx.x;
  sh[t] = v;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (t < s) { KS a = sh[t]; kcomb(a, sh[t + s]); sh[t] = a; }
    __syncthreads();
  }
  KS r = sh[0];
  __syncthreads();
  return r;
}

// The same for N quantities at once: shuffles inside the warps, then shuffles over
// the warps' pairs, so a block pays two barriers instead of
// a shared-memory tree per quantity (nine of them were 9 us of the 22 us that
// the diagnostics of a 32^3 box took). Thread d * THREADS / 32 returns quantity d.
template <int N, int THREADS>
__device__ __forceinline__ KS block_reduce_n(KS (&v)[N], KS (&sh)[THREADS / 32][N]) {
  static_assert(THREADS % 32 == 0 && N * (THREADS / 32) <= THREADS && 32 % (THREADS / 32) == 0, "whole warps");
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 0; d < N; ++d) {
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      const KS o = {__shfl_down_sync(0xffffffffu, v[d].s, s), __shfl_down_sync(0xffffffffu, v[d].c, s)};
      kcomb(v[d], o);
    }
    if (lane == 0) sh[w][d] = v[d];
  }
  __syncthreads();
  // W threads per quantity and a tree again: thread d * W returns quantity d
  constexpr int W = THREADS / 32;
  KS r = {0.0, 0.0};
  if (threadIdx.x < (N * W + 31) / 32 * 32) {
    if (threadIdx.x < N * W) r = sh[threadIdx.x % W][threadIdx.x / W];
#pragma unroll
    for (int s = W / 2; s > 0; s >>= 1) {
      const KS o = {__shfl_down_sync(0xffffffffu, r.s, s, W), __shfl_down_sync(0xffffffffu, r.c, s, W)};
      kcomb(r, o);
    }
  }
  return r;
}

}  // namespace bgk
