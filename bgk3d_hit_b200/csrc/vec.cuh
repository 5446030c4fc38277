// Row handling shared by the kernels that work on several cells of a row per
// thread: which lanes exchange x-neighbours, the x-shift of loaded chunks and
// the collision of packed FP16 cells.
#pragma once
#include "kernels.h"

namespace bgk {

__device__ __forceinline__ unsigned short u16_at(const __half* p) { return *reinterpret_cast<const unsigned short*>(p); }
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

// Place of a thread of a several-cells-per-thread kernel (V cells of a row per
// thread, 128-thread blocks over the ny*tpr threads of a plane).
// FLAT = false: nx/V = tpr is a power of two (arg = its logarithm) and ny*tpr a
// multiple of 32, so warps and rows are aligned with each other. FLAT = true:
// any nx, arg = tpr; row boundaries fall anywhere in a warp, the last chunk with
// cells may hold only `cells` < V of them, and chunks behind it (pad, where the
// launch asks for padded rows) work on the row's padding. Nothing in the
// padding ever reaches a cell.
template <int V, bool FLAT> struct VecPlace {
  int tpr, j, pos;
  int i0, i_prev, i_next;  // first cell, and the (periodic) elements before and behind the chunk
  int cells;               // cells of the row's last chunk
  bool valid;              // false: past the plane's last thread; j is clamped
  bool end;                // the row's last chunk with cells, or behind it
  __device__ VecPlace(const Geo& g, int arg) : VecPlace(g, arg, blockIdx.x * blockDim.x + threadIdx.x) {}
  // The same once more, so that nothing of it stays in registers in between (flat
  // rows: the aligned ones' decode is cheap to keep).
  __device__ VecPlace again(const Geo& g, int arg) const {
    if (!FLAT) return *this;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    asm volatile("" : "+r"(t));
    return VecPlace(g, arg, t);
  }
  __device__ VecPlace(const Geo& g, int arg, int t) {
    if (FLAT) {
      tpr = arg;
      j = (int)((unsigned)t / (unsigned)tpr);
      pos = t - j * tpr;
      const int e = (g.nx - 1) / V;
      cells = g.nx - V * e;
      end = pos >= e;
    } else {
      tpr = 1 << arg;
      j = t >> arg;
      pos = t & (tpr - 1);
      cells = V;
      end = pos == tpr - 1;
    }
    valid = j < g.ny;
    if (!valid) j = FLAT ? g.ny - 1 : 0;
    i0 = pos * V;
    i_prev = pos == 0 ? g.nx - 1 : i0 - 1;
    i_next = end ? 0 : i0 + V;
  }
  __device__ bool last() const { return FLAT && end && cells < V; }
};

// Lanes that exchange x-neighbours in the several-cells-per-thread kernels.
// Aligned rows shorter than a warp wrap inside it; rows of one or more warps
// wrap through global memory at the warp's first / last lane (edge_prev /
// edge_next). FLAT rows: the lanes at a row's ends are edges too.
struct XLanes {
  int src_prev, src_next;
  bool edge_prev, edge_next;
  template <int V, bool FLAT> __device__ XLanes(const VecPlace<V, FLAT>& at, int lane) {
    edge_prev = edge_next = false;
    if (FLAT || at.tpr >= 32) {
      src_prev = (lane + 31) & 31;
      src_next = (lane + 1) & 31;
      edge_prev = lane == 0 || (FLAT && at.pos == 0);
      edge_next = lane == 31 || (FLAT && at.end);
    } else {
      src_prev = at.pos == 0 ? lane + at.tpr - 1 : lane - 1;
      src_next = at.pos == at.tpr - 1 ? lane - at.tpr + 1 : lane + 1;
    }
  }
};

// Neighbouring warps of the block that an AA odd step's warp-edge lanes pass
// their crossing values to: prev_in / next_in where the row goes on in warp
// wprev / wnext of the same block.
struct EdgeWarps {
  bool any, prev_in, next_in;
  int wprev, wnext;
  template <int V, bool FLAT> __device__ explicit EdgeWarps(const VecPlace<V, FLAT>& at) {
    const int w = threadIdx.x >> 5;
    any = FLAT || at.tpr >= 32;
    prev_in = next_in = false;
    wprev = w - 1;
    wnext = w + 1;
    if (FLAT) {
      prev_in = w > 0 && at.pos != 0;
      next_in = w < 3 && !at.end;
    } else if (any) {
      const int nw = at.tpr >> 5, r = at.pos >> 5;  // warps per row, this warp's place in its row
      if (nw <= 4) {  // the whole row in this block
        prev_in = next_in = true;
        wprev = w - r + (r + nw - 1) % nw;
        wnext = w - r + (r + 1) % nw;
      } else {
        prev_in = w > 0;
        next_in = w < 3;
      }
    }
  }
};

// In a row's last chunk of `cells` cells, the element behind the last cell is
// the row's first one, which the lane loaded into E (pulls with cx < 0).
__device__ __forceinline__ void wrap_last(uint2 (&Y)[Q], const unsigned short (&E)[Q], int cells) {
#pragma unroll
  for (int q = 9; q < 14; ++q) {
    if (cells == 1) Y[q].x = __byte_perm(Y[q].x, E[q], 0x5410);
    else if (cells == 2) Y[q].y = __byte_perm(Y[q].y, E[q], 0x3254);
    else Y[q].y = __byte_perm(Y[q].y, E[q], 0x5410);
  }
}
__device__ __forceinline__ void wrap_last(float2 (&Y)[Q], const float (&E)[Q], int) {
#pragma unroll
  for (int q = 9; q < 14; ++q) Y[q].y = E[q];
}

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

// From how many cells the automatic choice takes the several-cells-per-thread
// kernels: below, their fewer and longer threads leave the chip idle and one
// cell per thread is faster. Measured us per step, one cell / several: AA FP16
// 32^3 4.1 / 5.1, 48^3 6.2 / 7.2, 210,000 cells 7.8 / 8.6, 64^3 7.7 / 7.2; FP32
// two-lattice 33^3 4.1 / 5.1, 48^3 6.2 / 6.2, 66^3 10.3 / 8.2.
constexpr long long VEC_MIN_TWO = 1LL << 17, VEC_MIN_AA = 1LL << 18;

// Rows of a V-cells-per-thread kernel: aligned (arg = log2(nx/V)) where nx/V is
// a power of two and a plane holds whole warps, else flat (arg = chunks of a
// row). padded: up to a 32-byte sector (8-byte chunks), for kernels that write
// rows they have not read: a partly written sector costs memory a read (FP16
// two-lattice step at 180^3:
// 74.3 GLUPS against 58.5 with rows cut at their last chunk, and 67 with zeros
// stored by lanes of their own; the AA step has read its rows and gains nothing). whole: only rows of whole chunks (the
// 16-byte kernels); arg < 0: not for them.
struct VecRows {
  bool flat;
  int arg, tpr;
  VecRows(const Geo& g, int V, bool padded, bool whole = false)
      : flat(true), arg(padded ? (g.nx + 4 * V - 1) / (4 * V) * 4 : (g.nx + V - 1) / V), tpr(arg) {
    if (whole && g.nx % V) {
      arg = -1;
      return;
    }
    const int t = g.nx / V;
    if (g.nx % V || (t & (t - 1)) || ((long long)g.ny * t) % 32) return;
    flat = false;
    tpr = t;
    arg = 0;
    while ((1 << arg) < tpr) ++arg;
  }
  // For the adjoint's steps and the interior of z-slabs (`planes` planes): aligned rows
  // at any size, others from VEC_MIN_TWO cells. us per step of bgk_adjoint's forward
  // run, FP32, one cell / two: 33^3 3.6 / 3.7, 40^3 4.15 / 5.0, 45^3 4.3 / 5.1, 50^3 4.2 /
  // 5.4, 56^3 5.8 / 5.8; two slabs of these sizes on one GPU are bound by the host's
  // calls (20 us a step either way).
  bool pays(const Geo& g, int planes) const { return !flat || (long long)g.nx * g.ny * planes >= VEC_MIN_TWO; }
};

}  // namespace bgk
