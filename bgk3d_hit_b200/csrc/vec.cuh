// Row handling shared by the kernels that work on several cells of a row per
// thread: which lanes exchange x-neighbours, the x-shift of loaded chunks and
// the collision of packed FP16 cells.
#pragma once
#include "kernels.h"

namespace bgk {

__device__ __forceinline__ unsigned short ldg_u16(const __half* p) {
  return __ldg(reinterpret_cast<const unsigned short*>(p));
}
__device__ __forceinline__ unsigned h2u(__half2 h) { return *reinterpret_cast<unsigned*>(&h); }
__device__ __forceinline__ float2 u2f2(unsigned u) { return __half22float2(*reinterpret_cast<__half2*>(&u)); }

// Collision of four FP16 cells packed in Y (population q of cell m in half m
// of Y[q]), F16::cell's arithmetic, on cells 0, 1 (low words) then cells 2, 3
// (high words): each half's outputs replace its inputs in Y, so only two
// cells' moments are live at a time. LES: the Smagorinsky collision
// (moments16_les: per-cell relaxation constants, the same pair update).
template <bool LES>
__device__ __forceinline__ void collide4_f16(uint2 (&Y)[Q], const StepK& K) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    Mom16 M[2];
    float om1[2] = {K.om1, K.om1};
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      float y[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const float2 f = u2f2(h ? Y[q].y : Y[q].x);
        y[q] = m ? f.y : f.x;
      }
      if constexpr (LES) M[m] = moments16_les(y, K, om1[m]);
      else M[m] = moments16(y, K);
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const int r = oppq(q);
      const float2 a = u2f2(h ? Y[q].y : Y[q].x), c = u2f2(h ? Y[r].y : Y[r].x);
      float p0, p1, o0, o1;
      pair16(q, a.x, c.x, M[0], om1[0], p0, o0);
      pair16(q, a.y, c.y, M[1], om1[1], p1, o1);
      const unsigned pq = h2u(__floats2half2_rn(p0, p1)), pr = h2u(__floats2half2_rn(o0, o1));
      if (h) { Y[q].y = pq; Y[r].y = pr; } else { Y[q].x = pq; Y[r].x = pr; }
    }
    {
      const float2 a = u2f2(h ? Y[Q - 1].y : Y[Q - 1].x);
      const unsigned pz = h2u(__floats2half2_rn(rest16(a.x, M[0], om1[0]), rest16(a.y, M[1], om1[1])));
      if (h) Y[Q - 1].y = pz; else Y[Q - 1].x = pz;
    }
  }
}

// Lanes that exchange x-neighbours in the several-cells-per-thread kernels:
// a row of nx cells is tpr = nx/V consecutive threads (V cells per thread).
// Rows shorter than a warp wrap inside it; rows of one or more warps wrap
// through global memory at the warp's first / last lane (edge_prev /
// edge_next).
struct XLanes {
  int src_prev, src_next;
  bool edge_prev, edge_next;
  __device__ XLanes(int tpr, int pos, int lane) {
    edge_prev = edge_next = false;
    if (tpr >= 32) {
      src_prev = (lane + 31) & 31;
      src_next = (lane + 1) & 31;
      edge_prev = lane == 0;
      edge_next = lane == 31;
    } else {
      src_prev = pos == 0 ? lane + tpr - 1 : lane - 1;
      src_next = pos == tpr - 1 ? lane - tpr + 1 : lane + 1;
    }
  }
};

// Second half of the x-shifted row loads of the four-cells-per-thread FP16
// kernels. Y[q] holds the aligned chunk of elements i0..i0+3 of population
// q's source row; cells i0..i0+3 need elements i0 - cx ... i0 + 3 - cx with
// cx = c_q,x, so the element that crosses the chunk boundary comes from the
// neighbouring lane (warp shuffle) or, for a warp's edge lane, from E[q],
// which that lane loaded together with the chunks. All loads are issued
// before the first shuffle: measured on B200 (FP16 AA odd step, 256^3), this
// ordering lifted the pair of AA steps from 72.2 to 75.6 GLUPS.
__device__ __forceinline__ void shift_rows(uint2 (&Y)[Q], const unsigned short (&E)[Q], const XLanes& xl) {
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const uint2 A = Y[q];
    if (cxq(q) > 0) {  // elements i0-1 .. i0+2
      unsigned prev = __shfl_sync(0xffffffffu, A.y >> 16, xl.src_prev);
      if (xl.edge_prev) prev = E[q];
      Y[q].x = __byte_perm(A.x, prev, 0x1054);
      Y[q].y = __byte_perm(A.x, A.y, 0x5432);
    } else if (cxq(q) < 0) {  // elements i0+1 .. i0+4
      unsigned next = __shfl_sync(0xffffffffu, A.x & 0xffffu, xl.src_next);
      if (xl.edge_next) next = E[q];
      Y[q].x = __byte_perm(A.x, A.y, 0x5432);
      Y[q].y = __byte_perm(A.y, next, 0x5432);
    }
  }
}

// Second half of the x-shifted row loads of the two-cells-per-thread FP32
// kernels: shift_rows on chunks of two floats (Y[q] holds elements i0, i0+1;
// the element that crosses the chunk comes from the neighbouring lane or, for
// a warp's edge lane, from E[q]).
__device__ __forceinline__ void shift_rows_f32(float2 (&Y)[Q], const float (&E)[Q], const XLanes& xl) {
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const float2 A = Y[q];
    if (cxq(q) > 0) {  // elements i0-1, i0
      float prev = __shfl_sync(0xffffffffu, A.y, xl.src_prev);
      if (xl.edge_prev) prev = E[q];
      Y[q] = make_float2(prev, A.x);
    } else if (cxq(q) < 0) {  // elements i0+1, i0+2
      float next = __shfl_sync(0xffffffffu, A.x, xl.src_next);
      if (xl.edge_next) next = E[q];
      Y[q] = make_float2(A.y, next);
    }
  }
}

// log2(nx/V) when a V-cells-per-thread kernel applies (nx/V a power of two,
// whole warps per plane), else -1.
inline int vec_log_tpr(const Geo& g, int V) {
  if (g.nx % V) return -1;
  const int tpr = g.nx / V;
  if (tpr & (tpr - 1)) return -1;
  if (((long long)g.ny * tpr) % 32) return -1;
  int l = 0;
  while ((1 << l) < tpr) ++l;
  return l;
}

}  // namespace bgk
