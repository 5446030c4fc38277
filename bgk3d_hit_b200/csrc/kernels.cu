// CUDA kernels of the BGK3D_HIT hot path for sm_100a.
//
//   k_two        fused pull-stream + BGK collide, two lattices, pop 19 in place
//                (SRC/col_MC.F90:98-421); periodic wrap by index arithmetic
//                replaces the halo exchange of SRC/bcond.comm.step3.F90
//   k_aa         in-place AA-pattern variant of the same update (no reference
//                counterpart; same per-cell arithmetic)
//   k_two_f32v, k_aa_f32v / k_two_f16v, k_aa_f16v
//                the same updates with two FP32 / four FP16 cells of a row per
//                thread (8-byte accesses, x-crossing values by warp shuffle);
//                the defaults of those forms from VEC_MIN_* cells
//   k_aa_f16w, k_aa_f32w
//                the AA odd step with eight FP16 (BGK) / four FP32 (BGK and
//                Smagorinsky) cells per thread, 16-byte accesses: its default
//                where rows are whole chunks
//   k_slab       two-lattice step of one z-slab with the face exchange fused in
//   k_init_*     equilibrium initial conditions (SRC/init.F90:83-141)
//   k_diag       diagno + dissipation + strain-rate sums (SRC/diagno.F90:73-121,
//                SRC/dissipation.F90:65-269) as deterministic compensated
//                per-block partials
//   k_enstrophy  0.5|curl u|^2 from the local velocity field
//   k_shift3     shift-only stencil of SRC/do_somethingGPU.F90:37-100
#include <algorithm>
#include <cmath>

#include "kernels.h"
#include "launch.cuh"
#include "reduce.cuh"
#include "vec.cuh"

namespace bgk {

__device__ __forceinline__ int wrapi(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// Read-only loads, for the kernels that no launch overlaps (see step_begin).
__device__ __forceinline__ double ldg(const double* p) { return __ldg(p); }
__device__ __forceinline__ float ldg(const float* p) { return __ldg(p); }
__device__ __forceinline__ __half ldg(const __half* p) { return __ldg(p); }

// Moments of 19 local deviations in the reference's order
// (SRC/diagno.F90:96-104, identical to SRC/col_MC.F90:133-141).
template <class V>
__device__ __forceinline__ V moments(const V (&x)[Q], V& vx, V& vy, V& vz) {
  using N = Num<V>;
  const V cte1 = N::c(1.0);
  V rho = x[0] + x[1] + x[2] + x[3] + x[4] + x[5] + x[6] + x[7]
        + x[8] + x[9] + x[10] + x[11] + x[12] + x[13] + x[14] + x[15]
        + x[16] + x[17] + x[18] + cte1;
  V rhoinv = ercp(rho);
  vx = (x[0] + x[1] + x[2] + x[3] + x[4] - x[9] - x[10] - x[11] - x[12] - x[13]) * rhoinv;
  vy = (x[2] + x[6] + x[7] + x[8] + x[11] - x[0] - x[9] - x[15] - x[16] - x[17]) * rhoinv;
  vz = (x[3] + x[5] + x[6] + x[12] + x[17] - x[1] - x[8] - x[10] - x[14] - x[15]) * rhoinv;
  return rho;
}

// Launch shape of the per-cell stream kernels: x-rows in blockDim.x.
struct Shape { dim3 grid, block; };
static Shape cell_shape(const Geo& g) {
  int tx = g.nx >= 128 ? 128 : ((g.nx + 31) / 32) * 32;
  int ty = 256 / tx;
  Shape s;
  s.block = dim3(tx, ty, 1);
  s.grid = dim3((g.nx + tx - 1) / tx, (g.ny + ty - 1) / ty, g.nz);
  return s;
}

static int grid_1d(long long n, int threads, int cap) {
  long long b = (n + threads - 1) / threads;
  return (int)(b < cap ? (b < 1 ? 1 : b) : cap);
}

// ------------------------------------------------------------- two lattice
template <class F, bool LES = false>
__global__ void __launch_bounds__(256) k_two(Pops<const typename F::S> src, Pops<typename F::S> dst, Geo g, StepK K) {
  step_begin();
  using S = typename F::S;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  // a row's threads run on to the end of its last 32-byte sector (padding, which
  // reaches no cell): a partly written sector costs memory a read
  constexpr int P = 32 / sizeof(S);
  if (i >= (g.nx + P - 1) / P * P || j >= g.ny) return;
  const int im = i == 0 ? g.nx - 1 : i - 1, ip = i >= g.nx - 1 ? 0 : i + 1;
  const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
  const int km = k == 0 ? g.nz - 1 : k - 1, kp = k == g.nz - 1 ? 0 : k + 1;
  S v[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    // pull from (i - cx, j - cy, k - cz), SRC/col_MC.F90:113-131
    const int ii = cxq(q) > 0 ? im : (cxq(q) < 0 ? ip : i);
    const int jj = cyq(q) > 0 ? jm : (cyq(q) < 0 ? jp : j);
    const int kk = czq(q) > 0 ? km : (czq(q) < 0 ? kp : k);
    const int off = ii + g.sx * (jj + g.ny * kk);
    // pop 19: in the time loop it is updated in place (src.p[18] == dst.p[18]); the
    // adjoint's out-of-place steps pass distinct arrays
    v[q] = src.p[q][off];
  }
  F::template cell<LES>(v, K);
  const int o = i + g.sx * (j + g.ny * k);
#pragma unroll
  for (int q = 0; q < Q; ++q) dst.p[q][o] = v[q];
}

// FP16 two-lattice step with 4 cells per thread and 8-byte accesses. A row of
// nx cells is handled by tpr consecutive threads (VecPlace).
// x-shifted pulls take the element that crosses a thread boundary from the
// neighbouring lane (warp shuffle); across warp boundaries (tpr > 32) lanes 0
// and 31 load it. Each cell's arithmetic is F16::cell's (moments16, pair16,
// rest16). The collision runs on two cells at a time, their outputs replacing
// their inputs in the packed registers, and the kernel runs 128-thread blocks
// at 96 registers (5 blocks per SM, no spills). On B200 at 256^3, with every
// row load issued before the shuffles, that measured 84.4 GLUPS against 82.0
// capped at 80 registers (6 blocks per SM, 52 spilled bytes; the Smagorinsky
// variant 78.5 against 67.9 with 108 spilled bytes); earlier forms of the
// kernel measured 76.6 with 256-thread blocks, 64.5 for all four cells at once
// at 2 blocks per SM and 58.4 at 64 registers (heavy spills).
template <bool LES, bool FLAT>
__global__ void __launch_bounds__(128, 5) k_two_f16v(Pops<const __half> src, Pops<__half> dst, Geo g, StepK K,
                                                  int rows, int k0) {
  step_begin();
  const VecPlace<4, FLAT> at(g, rows);
  const int k = blockIdx.y + k0;  // planes k0 .. k0 + gridDim.y - 1
  if (!at.valid) return;  // whole warps unless FLAT; no lane needs a value of theirs
  const XLanes xl(at, threadIdx.x & 31);
  const int j = at.j, i0 = at.i0;
  const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
  const int km = k == 0 ? g.nz - 1 : k - 1, kp = k == g.nz - 1 ? 0 : k + 1;
  uint2 Y[Q];  // four cells' stored values per population, cell m in half m
  unsigned short E[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int jj = cyq(q) > 0 ? jm : (cyq(q) < 0 ? jp : j);
    const int kk = czq(q) > 0 ? km : (czq(q) < 0 ? kp : k);
    const __half* p = (q == Q - 1 ? (const __half*)dst.p[Q - 1] : src.p[q]) + g.sx * (jj + g.ny * kk);
    Y[q] = *reinterpret_cast<const uint2*>(p + i0);
    E[q] = 0;
    if (cxq(q) > 0 && xl.edge_prev) E[q] = u16_at(p + at.i_prev);
    if (cxq(q) < 0 && xl.edge_next) E[q] = u16_at(p + at.i_next);
  }
  if (at.last()) wrap_last(Y, E, at.cells);
  shift_rows(Y, E, xl);
  collide4_f16<LES>(Y, K);
  const int o = i0 + g.sx * (j + g.ny * k);
#pragma unroll
  for (int q = 0; q < Q; ++q) *reinterpret_cast<uint2*>(dst.p[q] + o) = Y[q];
}

// FP32 two-lattice step with 2 cells per thread and 8-byte accesses (tpr =
// chunks of a row): k_two_f16v's row split and x-crossing shuffles on
// chunks of two floats, F32::cell's arithmetic on each cell, so the results
// are those of k_two<F32>. 72 registers (80 for the Smagorinsky step), no
// spills.
template <bool LES, bool FLAT>
__global__ void __launch_bounds__(128, 5) k_two_f32v(Pops<const float> src, Pops<float> dst, Geo g, StepK K,
                                                  int rows, int k0) {
  step_begin();
  const VecPlace<2, FLAT> at(g, rows);
  const int k = blockIdx.y + k0;  // planes k0 .. k0 + gridDim.y - 1
  if (!at.valid) return;  // whole warps unless FLAT; no lane needs a value of theirs
  const XLanes xl(at, threadIdx.x & 31);
  const int j = at.j, i0 = at.i0;
  const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
  const int km = k == 0 ? g.nz - 1 : k - 1, kp = k == g.nz - 1 ? 0 : k + 1;
  float2 Y[Q];  // two cells' values per population, cell m in component m
  float E[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int jj = cyq(q) > 0 ? jm : (cyq(q) < 0 ? jp : j);
    const int kk = czq(q) > 0 ? km : (czq(q) < 0 ? kp : k);
    // pop 19: updated in place in the time loop, distinct arrays in the adjoint's steps
    const float* p = src.p[q] + g.sx * (jj + g.ny * kk);
    Y[q] = *reinterpret_cast<const float2*>(p + i0);
    E[q] = 0.f;
    if (cxq(q) > 0 && xl.edge_prev) E[q] = *(p + at.i_prev);
    if (cxq(q) < 0 && xl.edge_next) E[q] = *(p + at.i_next);
  }
  if (at.last()) wrap_last(Y, E, at.cells);
  shift_rows_f32(Y, E, xl);
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    float s[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) s[q] = m ? Y[q].y : Y[q].x;
    F32::cell<LES>(s, K);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (m) Y[q].y = s[q];
      else Y[q].x = s[q];
    }
  }
  const int o = i0 + g.sx * (j + g.ny * k);
#pragma unroll
  for (int q = 0; q < Q; ++q) *reinterpret_cast<float2*>(dst.p[q] + o) = Y[q];
}

// FP16 two-lattice step with 2 cells per thread and 4-byte accesses (tpr =
// nx/2 threads per row); otherwise as k_two_f16v.
__global__ void __launch_bounds__(256, 4) k_two_f16v2(Pops<const __half> src, Pops<__half> dst, Geo g, StepK K,
                                                   int log_tpr) {
  step_begin();
  const int tpr = 1 << log_tpr;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = t >> log_tpr, pos = t & (tpr - 1);
  const int k = blockIdx.y;
  if (j >= g.ny) return;  // whole warps: ny*tpr is a multiple of 32
  const int lane = threadIdx.x & 31;
  const int i0 = pos * 2;
  const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
  const int km = k == 0 ? g.nz - 1 : k - 1, kp = k == g.nz - 1 ? 0 : k + 1;
  int src_prev, src_next;
  bool load_prev = false, load_next = false;
  if (tpr >= 32) {
    src_prev = (lane + 31) & 31;
    src_next = (lane + 1) & 31;
    load_prev = lane == 0;
    load_next = lane == 31;
  } else {
    src_prev = pos == 0 ? lane + tpr - 1 : lane - 1;
    src_next = pos == tpr - 1 ? lane - tpr + 1 : lane + 1;
  }
  const int i_prev = pos == 0 ? g.nx - 1 : i0 - 1;
  const int i_next = pos == tpr - 1 ? 0 : i0 + 2;
  unsigned Y[Q];  // two cells' stored values per population, cell m in half m
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int jj = cyq(q) > 0 ? jm : (cyq(q) < 0 ? jp : j);
    const int kk = czq(q) > 0 ? km : (czq(q) < 0 ? kp : k);
    const __half* p = (q == Q - 1 ? (const __half*)dst.p[Q - 1] : src.p[q]) + g.sx * (jj + g.ny * kk);
    const unsigned A = *reinterpret_cast<const unsigned*>(p + i0);
    if (cxq(q) == 0) {
      Y[q] = A;
    } else if (cxq(q) > 0) {  // cells need elements i0-1, i0
      unsigned prev = __shfl_sync(0xffffffffu, A >> 16, src_prev);
      if (load_prev) prev = u16_at(p + i_prev);
      Y[q] = __byte_perm(A, prev, 0x1054);
    } else {  // cells need elements i0+1, i0+2
      unsigned next = __shfl_sync(0xffffffffu, A & 0xffffu, src_next);
      if (load_next) next = u16_at(p + i_next);
      Y[q] = __byte_perm(A, next, 0x5432);
    }
  }
  Mom16 M[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    float y[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float2 f = u2f2(Y[q]);
      y[q] = m ? f.y : f.x;
    }
    M[m] = moments16(y, K);
  }
  const int o = i0 + g.sx * (j + g.ny * k);
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    const int r = oppq(q);
    const float2 a = u2f2(Y[q]), c = u2f2(Y[r]);
    float p0, p1, o0, o1;
    pair16(q, a.x, c.x, M[0], K.om1, p0, o0);
    pair16(q, a.y, c.y, M[1], K.om1, p1, o1);
    *reinterpret_cast<unsigned*>(dst.p[q] + o) = h2u(__floats2half2_rn(p0, p1));
    *reinterpret_cast<unsigned*>(dst.p[r] + o) = h2u(__floats2half2_rn(o0, o1));
  }
  {
    const float2 a = u2f2(Y[Q - 1]);
    *reinterpret_cast<unsigned*>(dst.p[Q - 1] + o) =
        h2u(__floats2half2_rn(rest16(a.x, M[0], K.om1), rest16(a.y, M[1], K.om1)));
  }
}

// --------------------------------------------------------------- AA pattern
// Even step: g_q(x) = slot q at x; result q -> slot opp(q) at x.
// Odd step:  g_q(x) = slot opp(q) at x - c_q; result q -> slot q at x + c_q.
// Each thread reads exactly the locations it writes, so the update is
// race-free in place; a location is never read after it has been written.
template <class F, bool ODD, bool LES>
__device__ __forceinline__ void aa_cell(Pops<typename F::S>& a, const Geo& g, const StepK& K) {
  using S = typename F::S;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z;
  if (i >= g.nx || j >= g.ny) return;
  int o = i + g.sx * (j + g.ny * k);
  const int im = i == 0 ? g.nx - 1 : i - 1, ip = i == g.nx - 1 ? 0 : i + 1;
  const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
  const int km = k == 0 ? g.nz - 1 : k - 1, kp = k == g.nz - 1 ? 0 : k + 1;
  S v[Q];
  int off[Q];  // location x - c_q (read, slot opp(q)) == location x + c_opp(q) (write, slot opp(q))
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int ii = cxq(q) > 0 ? im : (cxq(q) < 0 ? ip : i);
    const int jj = cyq(q) > 0 ? jm : (cyq(q) < 0 ? jp : j);
    const int kk = czq(q) > 0 ? km : (czq(q) < 0 ? kp : k);
    off[q] = ii + g.sx * (jj + g.ny * kk);
    v[q] = ODD ? a.p[oppq(q)][off[q]] : a.p[q][o];
  }
  F::template cell<LES>(v, K);
  // The stores go to the places of the loads. The offsets are kept through the
  // collision, not the 64-bit addresses, which the compiler would hold otherwise
  // (FP64 124 registers, Smagorinsky 136). GLUPS of the pair of steps at 256^3, addresses
  // kept / offsets recomputed / offsets kept: FP64 21.6 / 19.6 / 21.9, Smagorinsky 15.8 /
  // 19.6 / 20.9; FP32 40.1 / 39.2 / 41.5, Smagorinsky 35.4 / 40.5 / 38.3; FP16 51 / 62 /
  // 61.5, Smagorinsky 55 / 56.5 / 59.
  if (!ODD) asm volatile("" : "+r"(o));
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (ODD) asm volatile("" : "+r"(off[q]));
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (ODD) a.p[q][off[oppq(q)]] = v[q];
    else a.p[oppq(q)][o] = v[q];
  }
}

template <class F, bool ODD, bool LES = false>
__global__ void __launch_bounds__(256) k_aa(Pops<typename F::S> a, Geo g, StepK K) {
  step_begin();
  aa_cell<F, ODD, LES>(a, g, K);
}

// The FP16 odd step (BGK) is latency-bound on registers: capped at 48 (5
// blocks per SM) it measured 53.7 against 50.4 GLUPS uncapped for that step at
// 256^3 on B200, a few spilled bytes included.
__global__ void __launch_bounds__(256, 5) k_aa_f16_odd(Pops<__half> a, Geo g, StepK K) {
  step_begin();
  aa_cell<F16, true, false>(a, g, K);
}

// FP16 AA pattern with four cells per thread (the same row split, shuffles
// and collision as k_two_f16v). Even step: slot q at x -> slot opp(q) at x,
// 8-byte accesses, no exchange. Odd step: slot opp(q) at x - c_q -> slot q at
// x + c_q, with the x-crossing values moved between lanes on both the load and
// the store side; on the store side a warp-edge lane gets its crossing value
// from the neighbouring warp of the block through shared memory after a block
// barrier, so only block boundaries need partial stores (a warp edge with 2-
// and 4-byte stores costs about as much as the rest of the warp's stores of
// that population: 240 -> 223 us per 256^3 odd step, AA pair 77.1 -> 80.1
// GLUPS). Every (location, slot) pair is still read and written by the
// thread of the cell that owns it in the one-cell-per-thread kernel, or by a
// lane of the same warp after a shuffle that orders it behind the owner's
// loads, or by a lane of another warp of the block after the barrier that
// follows every warp's loads, so the in-place update stays race-free.
// 128-thread blocks at 96 registers (5 blocks per SM) like k_two_f16v. The odd step stores to the
// rows it loaded from; left alone, the compiler keeps those 18 row addresses
// live through the collision, so the BGK odd step recomputes them from an
// opaque copy of (j, k) and fits 96 registers without spills (5 blocks per
// SM). On B200 at 256^3 the pair of steps measured 72.3 GLUPS, against 71.1
// with the addresses kept (128 registers, 4 blocks), 69.5 with 256-thread
// blocks, 63.4 with the odd step capped at 80 registers (282 spilled bytes),
// 62.8-65.0 with two cells per thread on the odd step, and 58 for one cell per
// thread; with the loads issued before the shuffles and the even step at 96
// registers as well, 76.9. The LES odd step recomputes its store rows the
// same way (96 registers, a few spilled bytes).
// Store side of the AA odd step: stores four cells' values Y (cells
// i0..i0+3) at elements i0 + cx ... i0 + 3 + cx of row p as one aligned
// 8-byte chunk, completed with the neighbouring lane's crossing value (warp
// shuffle). A warp-edge lane takes that value from the neighbouring warp
// through shared memory (from_prev / from_next) when that warp is in the same
// block (prev_in / next_in) and stores its whole chunk, the neighbour then
// skipping its store of the crossing element; at block boundaries the edge
// lanes store their part of the chunk and their crossing value with 4- and
// 2-byte stores.
template <bool FLAT>
__device__ __forceinline__ void shift_out(uint2 Y, int cx, __half* p, const VecPlace<4, FLAT>& at, const XLanes& xl,
                                          const EdgeWarps& ew, unsigned from_prev, unsigned from_next) {
  const int i0 = at.i0;
  unsigned short* u = reinterpret_cast<unsigned short*>(p);
  if (cx == 0) {
    *reinterpret_cast<uint2*>(p + i0) = Y;
  } else if (cx > 0) {  // cell i0+m -> element i0+m+1
    unsigned prev = __shfl_sync(0xffffffffu, Y.y >> 16, xl.src_prev);  // cell i0-1 of the lane before
    if (xl.edge_prev && ew.prev_in) prev = from_prev;
    const unsigned lo = __byte_perm(prev, Y.x, 0x5410), hi = __byte_perm(Y.x, Y.y, 0x5432);
    if (!xl.edge_prev || ew.prev_in) {
      *reinterpret_cast<uint2*>(p + i0) = make_uint2(lo, hi);
    } else {
      u[i0 + 1] = (unsigned short)(Y.x & 0xffffu);
      *reinterpret_cast<unsigned*>(p + i0 + 2) = hi;
    }
    if (xl.edge_next && !ew.next_in) {
      unsigned v = Y.y >> 16;
      if (at.last()) v = at.cells == 1 ? Y.x : (at.cells == 2 ? Y.x >> 16 : Y.y);
      u[at.i_next] = (unsigned short)(v & 0xffffu);
    }
  } else {  // cell i0+m -> element i0+m-1
    unsigned next = __shfl_sync(0xffffffffu, Y.x & 0xffffu, xl.src_next);  // cell i0+4 of the lane after
    if (xl.edge_next && ew.next_in) next = from_next;
    const unsigned lo = __byte_perm(Y.x, Y.y, 0x5432), hi = __byte_perm(Y.y, next, 0x5432);
    if (!xl.edge_next || ew.next_in) {
      *reinterpret_cast<uint2*>(p + i0) = make_uint2(lo, hi);
    } else if (at.last()) {
      // cells 1.. go one element back; the row's last element is its first cell's
      if (at.cells > 1) u[i0] = (unsigned short)(Y.x >> 16);
      if (at.cells > 2) u[i0 + 1] = (unsigned short)(Y.y & 0xffffu);
    } else {
      *reinterpret_cast<unsigned*>(p + i0) = lo;
      u[i0 + 2] = (unsigned short)(Y.y >> 16);
    }
    if (xl.edge_prev && !ew.prev_in) u[at.i_prev] = (unsigned short)(Y.x & 0xffffu);
  }
}

template <bool ODD, bool LES, bool FLAT>
__global__ void __launch_bounds__(128, 5) k_aa_f16v(Pops<__half> a, Geo g, StepK K, int rows) {
  step_begin();
  const VecPlace<4, FLAT> at(g, rows);
  const int k = blockIdx.y;
  const bool valid = at.valid;  // whole warps unless FLAT
  if (!ODD && !valid) return;
  const int j = at.j;  // idle threads of the odd step only reach its barrier
  const XLanes xl(at, threadIdx.x & 31);
  const int i0 = at.i0;
  const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
  const int km = k == 0 ? g.nz - 1 : k - 1, kp = k == g.nz - 1 ? 0 : k + 1;
  auto row = [&](int dy, int dz) {  // row offset of (j + dy, k + dz), dy, dz in {-1, 0, 1}
    const int jj = dy > 0 ? jp : (dy < 0 ? jm : j);
    const int kk = dz > 0 ? kp : (dz < 0 ? km : k);
    return g.sx * (jj + g.ny * kk);
  };
  uint2 Y[Q];
  if (ODD && !FLAT && !valid) {
#pragma unroll
    for (int q = 0; q < Q; ++q) Y[q] = make_uint2(0u, 0u);
  } else if (ODD) {
    unsigned short E[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const __half* p = a.p[oppq(q)] + row(-cyq(q), -czq(q));
      Y[q] = *reinterpret_cast<const uint2*>(p + i0);
      E[q] = 0;
      if (cxq(q) > 0 && xl.edge_prev) E[q] = u16_at(p + at.i_prev);
      if (cxq(q) < 0 && xl.edge_next) E[q] = u16_at(p + at.i_next);
    }
    if (at.last()) wrap_last(Y, E, at.cells);
    shift_rows(Y, E, xl);
  } else {
#pragma unroll
    for (int q = 0; q < Q; ++q) Y[q] = *reinterpret_cast<const uint2*>(a.p[q] + row(0, 0) + i0);
  }
  if (FLAT || valid) collide4_f16<LES>(Y, K);
  // odd step: the warps' crossing values (cx > 0 populations: the last
  // lane's last cell; cx < 0: the first lane's first cell) through shared
  // memory; the barrier also orders every warp's loads before any warp's
  // stores of its neighbours' crossing elements
  __shared__ unsigned xs_last[ODD ? 4 : 1][5], xs_first[ODD ? 4 : 1][5];
  const EdgeWarps ew(at);
  if (ODD) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (ew.any) {
      if (valid && lane == 31) {
#pragma unroll
        for (int q = 0; q < 5; ++q) xs_last[w][q] = Y[q].y >> 16;
      }
      if (valid && lane == 0) {
#pragma unroll
        for (int q = 9; q < 14; ++q) xs_first[w][q - 9] = Y[q].x & 0xffffu;
      }
    }
    __syncthreads();
    if (!valid) return;
  }
  const auto as = at.again(g, rows);
  const XLanes xs = FLAT ? XLanes(as, threadIdx.x & 31) : xl;
  const EdgeWarps es = FLAT ? EdgeWarps(as) : ew;
  int js = FLAT ? as.j : j, ks = k;  // store rows: recomputed after the collision
  asm volatile("" : "+r"(js), "+r"(ks));
  const int jms = js == 0 ? g.ny - 1 : js - 1, jps = js == g.ny - 1 ? 0 : js + 1;
  const int kms = ks == 0 ? g.nz - 1 : ks - 1, kps = ks == g.nz - 1 ? 0 : ks + 1;
  auto row_out = [&](int dy, int dz) {
    const int jj = dy > 0 ? jps : (dy < 0 ? jms : js);
    const int kk = dz > 0 ? kps : (dz < 0 ? kms : ks);
    return g.sx * (jj + g.ny * kk);
  };
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (!ODD) {
      *reinterpret_cast<uint2*>(a.p[oppq(q)] + row_out(0, 0) + i0) = Y[q];
    } else {
      const unsigned fp = cxq(q) > 0 && xs.edge_prev && es.prev_in ? xs_last[es.wprev][q] : 0u;
      const unsigned fn = cxq(q) < 0 && xs.edge_next && es.next_in ? xs_first[es.wnext][q - 9] : 0u;
      shift_out(Y[q], cxq(q), a.p[q] + row_out(cyq(q), czq(q)), as, xs, es, fp, fn);
    }
  }
}

// FP16 AA pattern with eight cells per thread: k_aa_f16v's structure on
// 16-byte chunks (cells i0..i0+7, i0 = 8 pos, tpr = nx/8 threads per row), so
// the per-thread work of the odd step's x-crossing (shuffles, warp-edge
// values, the 18 shifted rows' addresses) is spread over twice the cells.
// Per-cell arithmetic is collide4_f16's on each half of the chunk, so the
// results are k_aa_f16v's. The odd instantiation is launched (128
// registers, 4 blocks/SM); the even one measured no faster than k_aa_f16v.
__device__ __forceinline__ void shift_rows8(uint4 (&Y)[Q], const unsigned short (&E)[Q], const XLanes& xl) {
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const uint4 A = Y[q];
    if (cxq(q) > 0) {  // elements i0-1 .. i0+6
      unsigned prev = __shfl_sync(0xffffffffu, A.w >> 16, xl.src_prev);
      if (xl.edge_prev) prev = E[q];
      Y[q].x = __byte_perm(A.x, prev, 0x1054);
      Y[q].y = __byte_perm(A.x, A.y, 0x5432);
      Y[q].z = __byte_perm(A.y, A.z, 0x5432);
      Y[q].w = __byte_perm(A.z, A.w, 0x5432);
    } else if (cxq(q) < 0) {  // elements i0+1 .. i0+8
      unsigned next = __shfl_sync(0xffffffffu, A.x & 0xffffu, xl.src_next);
      if (xl.edge_next) next = E[q];
      Y[q].x = __byte_perm(A.x, A.y, 0x5432);
      Y[q].y = __byte_perm(A.y, A.z, 0x5432);
      Y[q].z = __byte_perm(A.z, A.w, 0x5432);
      Y[q].w = __byte_perm(A.w, next, 0x5432);
    }
  }
}

// Store side of the eight-cells odd step (shift_out on 16-byte chunks): cell
// i0+m goes to element i0+m+cx; the aligned chunk i0..i0+7 is completed with
// the neighbouring lane's crossing value, and at block boundaries the edge
// lanes store their part with 2-, 4- and 8-byte stores.
template <bool FLAT>
__device__ __forceinline__ void shift_out8(uint4 Y, int cx, __half* p, const VecPlace<8, FLAT>& at, const XLanes& xl,
                                           const EdgeWarps& ew, unsigned from_prev, unsigned from_next) {
  const int i0 = at.i0;
  unsigned short* u = reinterpret_cast<unsigned short*>(p);
  if (cx == 0) {
    *reinterpret_cast<uint4*>(p + i0) = Y;
  } else if (cx > 0) {  // cell i0+m -> element i0+m+1
    unsigned prev = __shfl_sync(0xffffffffu, Y.w >> 16, xl.src_prev);  // cell i0-1 of the lane before
    if (xl.edge_prev && ew.prev_in) prev = from_prev;
    const uint4 c = make_uint4(__byte_perm(prev, Y.x, 0x5410), __byte_perm(Y.x, Y.y, 0x5432),
                               __byte_perm(Y.y, Y.z, 0x5432), __byte_perm(Y.z, Y.w, 0x5432));
    if (!xl.edge_prev || ew.prev_in) {
      *reinterpret_cast<uint4*>(p + i0) = c;
    } else {
      u[i0 + 1] = (unsigned short)(Y.x & 0xffffu);
      *reinterpret_cast<unsigned*>(p + i0 + 2) = c.y;
      *reinterpret_cast<uint2*>(p + i0 + 4) = make_uint2(c.z, c.w);
    }
    if (xl.edge_next && !ew.next_in) u[at.i_next] = (unsigned short)(Y.w >> 16);
  } else {  // cell i0+m -> element i0+m-1
    unsigned next = __shfl_sync(0xffffffffu, Y.x & 0xffffu, xl.src_next);  // cell i0+8 of the lane after
    if (xl.edge_next && ew.next_in) next = from_next;
    const uint4 c = make_uint4(__byte_perm(Y.x, Y.y, 0x5432), __byte_perm(Y.y, Y.z, 0x5432),
                               __byte_perm(Y.z, Y.w, 0x5432), __byte_perm(Y.w, next, 0x5432));
    if (!xl.edge_next || ew.next_in) {
      *reinterpret_cast<uint4*>(p + i0) = c;
    } else {
      *reinterpret_cast<uint2*>(p + i0) = make_uint2(c.x, c.y);
      *reinterpret_cast<unsigned*>(p + i0 + 4) = c.z;
      u[i0 + 6] = (unsigned short)(Y.w >> 16);
    }
    if (xl.edge_prev && !ew.prev_in) u[at.i_prev] = (unsigned short)(Y.x & 0xffffu);
  }
}

template <bool ODD, bool FLAT>
__global__ void __launch_bounds__(128, 4) k_aa_f16w(Pops<__half> a, Geo g, StepK K, int rows) {
  step_begin();
  const VecPlace<8, FLAT> at(g, rows);
  const int k = blockIdx.y;
  const bool valid = at.valid;  // whole warps unless FLAT
  if (!ODD && !valid) return;
  const int j = at.j;  // idle threads of the odd step only reach its barrier
  const XLanes xl(at, threadIdx.x & 31);
  const int i0 = at.i0;
  const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
  const int km = k == 0 ? g.nz - 1 : k - 1, kp = k == g.nz - 1 ? 0 : k + 1;
  auto row = [&](int dy, int dz) {
    const int jj = dy > 0 ? jp : (dy < 0 ? jm : j);
    const int kk = dz > 0 ? kp : (dz < 0 ? km : k);
    return g.sx * (jj + g.ny * kk);
  };
  uint4 Y[Q];
  if (ODD && !FLAT && !valid) {
#pragma unroll
    for (int q = 0; q < Q; ++q) Y[q] = make_uint4(0u, 0u, 0u, 0u);
  } else if (ODD) {
    unsigned short E[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const __half* p = a.p[oppq(q)] + row(-cyq(q), -czq(q));
      Y[q] = *reinterpret_cast<const uint4*>(p + i0);
      E[q] = 0;
      if (cxq(q) > 0 && xl.edge_prev) E[q] = u16_at(p + at.i_prev);
      if (cxq(q) < 0 && xl.edge_next) E[q] = u16_at(p + at.i_next);
    }
    shift_rows8(Y, E, xl);
  } else {
#pragma unroll
    for (int q = 0; q < Q; ++q) Y[q] = *reinterpret_cast<const uint4*>(a.p[q] + row(0, 0) + i0);
  }
  if (FLAT || valid) {
    uint2 L[Q], H[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      L[q] = make_uint2(Y[q].x, Y[q].y);
      H[q] = make_uint2(Y[q].z, Y[q].w);
    }
    collide4_f16<false>(L, K);
    collide4_f16<false>(H, K);
#pragma unroll
    for (int q = 0; q < Q; ++q) Y[q] = make_uint4(L[q].x, L[q].y, H[q].x, H[q].y);
  }
  __shared__ unsigned xs_last[ODD ? 4 : 1][5], xs_first[ODD ? 4 : 1][5];
  const EdgeWarps ew(at);
  if (ODD) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (ew.any) {
      if (valid && lane == 31) {
#pragma unroll
        for (int q = 0; q < 5; ++q) xs_last[w][q] = Y[q].w >> 16;
      }
      if (valid && lane == 0) {
#pragma unroll
        for (int q = 9; q < 14; ++q) xs_first[w][q - 9] = Y[q].x & 0xffffu;
      }
    }
    __syncthreads();
    if (!valid) return;
  }
  const auto as = at.again(g, rows);
  const XLanes xs = FLAT ? XLanes(as, threadIdx.x & 31) : xl;
  const EdgeWarps es = FLAT ? EdgeWarps(as) : ew;
  int js = FLAT ? as.j : j, ks = k;
  asm volatile("" : "+r"(js), "+r"(ks));
  const int jms = js == 0 ? g.ny - 1 : js - 1, jps = js == g.ny - 1 ? 0 : js + 1;
  const int kms = ks == 0 ? g.nz - 1 : ks - 1, kps = ks == g.nz - 1 ? 0 : ks + 1;
  auto row_out = [&](int dy, int dz) {
    const int jj = dy > 0 ? jps : (dy < 0 ? jms : js);
    const int kk = dz > 0 ? kps : (dz < 0 ? kms : ks);
    return g.sx * (jj + g.ny * kk);
  };
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (!ODD) {
      *reinterpret_cast<uint4*>(a.p[oppq(q)] + row_out(0, 0) + i0) = Y[q];
    } else {
      const unsigned fp = cxq(q) > 0 && xs.edge_prev && es.prev_in ? xs_last[es.wprev][q] : 0u;
      const unsigned fn = cxq(q) < 0 && xs.edge_next && es.next_in ? xs_first[es.wnext][q - 9] : 0u;
      shift_out8(Y[q], cxq(q), a.p[q] + row_out(cyq(q), czq(q)), as, xs, es, fp, fn);
    }
  }
}

// Store side of the FP32 odd step: cells i0, i0+1 go to elements i0 + cx,
// i0 + 1 + cx of row p, stored as the aligned chunk (i0, i0+1) completed with
// the neighbouring lane's crossing value, as shift_out does for FP16.
template <bool FLAT>
__device__ __forceinline__ void shift_out_f32(float2 Y, int cx, float* p, const VecPlace<2, FLAT>& at, const XLanes& xl,
                                              const EdgeWarps& ew, float from_prev, float from_next) {
  const int i0 = at.i0;
  if (cx == 0) {
    *reinterpret_cast<float2*>(p + i0) = Y;
  } else if (cx > 0) {  // cell i0+m -> element i0+m+1
    float prev = __shfl_sync(0xffffffffu, Y.y, xl.src_prev);  // cell i0-1 of the lane before
    if (xl.edge_prev && ew.prev_in) prev = from_prev;
    if (!xl.edge_prev || ew.prev_in) *reinterpret_cast<float2*>(p + i0) = make_float2(prev, Y.x);
    else p[i0 + 1] = Y.x;
    if (xl.edge_next && !ew.next_in) p[at.i_next] = at.last() ? Y.x : Y.y;
  } else {  // cell i0+m -> element i0+m-1
    float next = __shfl_sync(0xffffffffu, Y.x, xl.src_next);  // cell i0+2 of the lane after
    if (xl.edge_next && ew.next_in) next = from_next;
    if (!xl.edge_next || ew.next_in) *reinterpret_cast<float2*>(p + i0) = make_float2(Y.y, next);
    else if (!at.last()) p[i0] = Y.y;
    if (xl.edge_prev && !ew.prev_in) p[at.i_prev] = Y.x;
  }
}

// FP32 AA pattern with two cells per thread: k_aa_f16v's row split (tpr =
// nx/2 threads per row), x-crossing shuffles and block-local warp-edge stores
// on 8-byte chunks of two floats, F32::cell's arithmetic (the reference's
// order) on each cell, so the results are those of k_aa<F32, ODD>. The same
// ownership argument keeps the in-place update race-free. 95 registers (87
// for the Smagorinsky even step), no spills.
template <bool ODD, bool LES, bool FLAT>
__global__ void __launch_bounds__(128, 5) k_aa_f32v(Pops<float> a, Geo g, StepK K, int rows) {
  step_begin();
  const VecPlace<2, FLAT> at(g, rows);
  const int k = blockIdx.y;
  const bool valid = at.valid;  // whole warps unless FLAT
  if (!ODD && !valid) return;
  const int j = at.j;  // idle threads of the odd step only reach its barrier
  const XLanes xl(at, threadIdx.x & 31);
  const int i0 = at.i0;
  const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
  const int km = k == 0 ? g.nz - 1 : k - 1, kp = k == g.nz - 1 ? 0 : k + 1;
  auto row = [&](int dy, int dz) {  // row offset of (j + dy, k + dz), dy, dz in {-1, 0, 1}
    const int jj = dy > 0 ? jp : (dy < 0 ? jm : j);
    const int kk = dz > 0 ? kp : (dz < 0 ? km : k);
    return g.sx * (jj + g.ny * kk);
  };
  float2 Y[Q];
  if (ODD && !FLAT && !valid) {
#pragma unroll
    for (int q = 0; q < Q; ++q) Y[q] = make_float2(0.f, 0.f);
  } else if (ODD) {
    float E[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float* p = a.p[oppq(q)] + row(-cyq(q), -czq(q));
      Y[q] = *reinterpret_cast<const float2*>(p + i0);
      E[q] = 0.f;
      if (cxq(q) > 0 && xl.edge_prev) E[q] = *(p + at.i_prev);
      if (cxq(q) < 0 && xl.edge_next) E[q] = *(p + at.i_next);
    }
    if (at.last()) wrap_last(Y, E, at.cells);
    shift_rows_f32(Y, E, xl);
  } else {
#pragma unroll
    for (int q = 0; q < Q; ++q) Y[q] = *reinterpret_cast<const float2*>(a.p[q] + row(0, 0) + i0);
  }
  if (FLAT || valid) {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      float s[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) s[q] = m ? Y[q].y : Y[q].x;
      F32::cell<LES>(s, K);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (m) Y[q].y = s[q];
        else Y[q].x = s[q];
      }
    }
  }
  __shared__ float xs_last[ODD ? 4 : 1][5], xs_first[ODD ? 4 : 1][5];
  const EdgeWarps ew(at);
  if (ODD) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (ew.any) {
      if (valid && lane == 31) {
#pragma unroll
        for (int q = 0; q < 5; ++q) xs_last[w][q] = Y[q].y;
      }
      if (valid && lane == 0) {
#pragma unroll
        for (int q = 9; q < 14; ++q) xs_first[w][q - 9] = Y[q].x;
      }
    }
    __syncthreads();
    if (!valid) return;
  }
  int js = j, ks = k;  // store rows: recomputed after the collision
  asm volatile("" : "+r"(js), "+r"(ks));
  const int jms = js == 0 ? g.ny - 1 : js - 1, jps = js == g.ny - 1 ? 0 : js + 1;
  const int kms = ks == 0 ? g.nz - 1 : ks - 1, kps = ks == g.nz - 1 ? 0 : ks + 1;
  auto row_out = [&](int dy, int dz) {
    const int jj = dy > 0 ? jps : (dy < 0 ? jms : js);
    const int kk = dz > 0 ? kps : (dz < 0 ? kms : ks);
    return g.sx * (jj + g.ny * kk);
  };
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (!ODD) {
      *reinterpret_cast<float2*>(a.p[oppq(q)] + row_out(0, 0) + i0) = Y[q];
    } else {
      const float fp = cxq(q) > 0 && xl.edge_prev && ew.prev_in ? xs_last[ew.wprev][q] : 0.f;
      const float fn = cxq(q) < 0 && xl.edge_next && ew.next_in ? xs_first[ew.wnext][q - 9] : 0.f;
      shift_out_f32(Y[q], cxq(q), a.p[q] + row_out(cyq(q), czq(q)), at, xl, ew, fp, fn);
    }
  }
}

// FP32 AA odd step with four cells per thread: k_aa_f32v's odd step on
// 16-byte chunks of four floats (cells i0..i0+3, i0 = 4 pos, tpr = nx/4), so
// its per-thread x-crossing work covers twice the cells, as k_aa_f16w does
// for FP16. F32::cell's arithmetic on each cell: the results of k_aa<F32>.
// 125 registers (127 with the Smagorinsky collision), 4 blocks/SM, no spills.
template <bool FLAT>
__device__ __forceinline__ void shift_out4_f32(float4 Y, int cx, float* p, const VecPlace<4, FLAT>& at, const XLanes& xl,
                                               const EdgeWarps& ew, float from_prev, float from_next) {
  const int i0 = at.i0;
  if (cx == 0) {
    *reinterpret_cast<float4*>(p + i0) = Y;
  } else if (cx > 0) {  // cell i0+m -> element i0+m+1
    float prev = __shfl_sync(0xffffffffu, Y.w, xl.src_prev);  // cell i0-1 of the lane before
    if (xl.edge_prev && ew.prev_in) prev = from_prev;
    if (!xl.edge_prev || ew.prev_in) {
      *reinterpret_cast<float4*>(p + i0) = make_float4(prev, Y.x, Y.y, Y.z);
    } else {
      p[i0 + 1] = Y.x;
      *reinterpret_cast<float2*>(p + i0 + 2) = make_float2(Y.y, Y.z);
    }
    if (xl.edge_next && !ew.next_in) p[at.i_next] = Y.w;
  } else {  // cell i0+m -> element i0+m-1
    float next = __shfl_sync(0xffffffffu, Y.x, xl.src_next);  // cell i0+4 of the lane after
    if (xl.edge_next && ew.next_in) next = from_next;
    if (!xl.edge_next || ew.next_in) {
      *reinterpret_cast<float4*>(p + i0) = make_float4(Y.y, Y.z, Y.w, next);
    } else {
      *reinterpret_cast<float2*>(p + i0) = make_float2(Y.y, Y.z);
      p[i0 + 2] = Y.w;
    }
    if (xl.edge_prev && !ew.prev_in) p[at.i_prev] = Y.x;
  }
}

template <bool LES, bool FLAT>
__global__ void __launch_bounds__(128, 4) k_aa_f32w(Pops<float> a, Geo g, StepK K, int rows) {
  step_begin();
  const VecPlace<4, FLAT> at(g, rows);
  const int k = blockIdx.y;
  const bool valid = at.valid;  // whole warps unless FLAT
  const int j = at.j;  // idle threads of the odd step only reach its barrier
  const XLanes xl(at, threadIdx.x & 31);
  const int i0 = at.i0;
  const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
  const int km = k == 0 ? g.nz - 1 : k - 1, kp = k == g.nz - 1 ? 0 : k + 1;
  auto row = [&](int dy, int dz) {
    const int jj = dy > 0 ? jp : (dy < 0 ? jm : j);
    const int kk = dz > 0 ? kp : (dz < 0 ? km : k);
    return g.sx * (jj + g.ny * kk);
  };
  float4 Y[Q];
  if (!FLAT && !valid) {
#pragma unroll
    for (int q = 0; q < Q; ++q) Y[q] = make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    float E[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float* p = a.p[oppq(q)] + row(-cyq(q), -czq(q));
      Y[q] = *reinterpret_cast<const float4*>(p + i0);
      E[q] = 0.f;
      if (cxq(q) > 0 && xl.edge_prev) E[q] = *(p + at.i_prev);
      if (cxq(q) < 0 && xl.edge_next) E[q] = *(p + at.i_next);
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float4 A = Y[q];
      if (cxq(q) > 0) {  // elements i0-1 .. i0+2
        float prev = __shfl_sync(0xffffffffu, A.w, xl.src_prev);
        if (xl.edge_prev) prev = E[q];
        Y[q] = make_float4(prev, A.x, A.y, A.z);
      } else if (cxq(q) < 0) {  // elements i0+1 .. i0+4
        float next = __shfl_sync(0xffffffffu, A.x, xl.src_next);
        if (xl.edge_next) next = E[q];
        Y[q] = make_float4(A.y, A.z, A.w, next);
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      float s[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) s[q] = m == 0 ? Y[q].x : (m == 1 ? Y[q].y : (m == 2 ? Y[q].z : Y[q].w));
      F32::cell<LES>(s, K);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (m == 0) Y[q].x = s[q];
        else if (m == 1) Y[q].y = s[q];
        else if (m == 2) Y[q].z = s[q];
        else Y[q].w = s[q];
      }
    }
  }
  __shared__ float xs_last[4][5], xs_first[4][5];
  const EdgeWarps ew(at);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (ew.any) {
    if (valid && lane == 31) {
#pragma unroll
      for (int q = 0; q < 5; ++q) xs_last[w][q] = Y[q].w;
    }
    if (valid && lane == 0) {
#pragma unroll
      for (int q = 9; q < 14; ++q) xs_first[w][q - 9] = Y[q].x;
    }
  }
  __syncthreads();
  if (!valid) return;
  int js = j, ks = k;  // store rows: recomputed after the collision
  asm volatile("" : "+r"(js), "+r"(ks));
  const int jms = js == 0 ? g.ny - 1 : js - 1, jps = js == g.ny - 1 ? 0 : js + 1;
  const int kms = ks == 0 ? g.nz - 1 : ks - 1, kps = ks == g.nz - 1 ? 0 : ks + 1;
  auto row_out = [&](int dy, int dz) {
    const int jj = dy > 0 ? jps : (dy < 0 ? jms : js);
    const int kk = dz > 0 ? kps : (dz < 0 ? kms : ks);
    return g.sx * (jj + g.ny * kk);
  };
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const float fp = cxq(q) > 0 && xl.edge_prev && ew.prev_in ? xs_last[ew.wprev][q] : 0.f;
    const float fn = cxq(q) < 0 && xl.edge_next && ew.next_in ? xs_first[ew.wnext][q - 9] : 0.f;
    shift_out4_f32(Y[q], cxq(q), a.p[q] + row_out(cyq(q), czq(q)), at, xl, ew, fp, fn);
  }
}

// ----------------------------------------------------------------- z-slabs
// Two-lattice step of one z-slab of a box split along z (the reference's
// proc_z ranks, SRC/setup_MPI.F90:112-131). x and y wrap in the kernel; a pull
// across a z face reads this slab's ghost plane instead of wrapping. The
// boundary planes' post-collision populations that cross a face are also
// stored straight into the neighbour's ghost plane for the next step (a peer
// store over NVLink when the neighbour is another GPU): the halo exchange of
// SRC/bcond.comm.step3.F90:77-297 fused into the producing kernel.
// EDGE = false: the interior planes 1..nz-2 (blockIdx.z + 1), whose pulls stay
// inside the slab (the whole-box kernel's code without the z wrap); EDGE =
// true: planes 0 and nz-1 (blockIdx.z = 0, 1), which read ghost planes and
// feed the neighbours. Separate kernels keep the interior one's registers
// (and so its occupancy) those of the whole-box kernel.
template <class F, bool LES, bool EDGE>
__global__ void __launch_bounds__(256) k_slab(Pops<const typename F::S> src, Pops<typename F::S> dst, Geo g,
                                              StepK K, Halo<typename F::S> h) {
  using S = typename F::S;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = EDGE ? (blockIdx.z == 0 ? 0 : g.nz - 1) : (int)blockIdx.z + 1;
  const bool active = i < g.nx && j < g.ny;
  if (!EDGE && !active) return;
  if (active) {
    const int im = i == 0 ? g.nx - 1 : i - 1, ip = i == g.nx - 1 ? 0 : i + 1;
    const int jm = j == 0 ? g.ny - 1 : j - 1, jp = j == g.ny - 1 ? 0 : j + 1;
    S v[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int ii = cxq(q) > 0 ? im : (cxq(q) < 0 ? ip : i);
      const int jj = cyq(q) > 0 ? jm : (cyq(q) < 0 ? jp : j);
      const int po = ii + g.sx * jj;
      if (EDGE && czq(q) > 0 && k == 0) v[q] = ldg(h.in_lo[zslot(q)] + po);
      else if (EDGE && czq(q) < 0 && k == g.nz - 1) v[q] = ldg(h.in_hi[zslot(q)] + po);
      else {
        const int off = po + g.sx * g.ny * (k - czq(q));
        v[q] = (q == Q - 1) ? src.p[Q - 1][off] : ldg(src.p[q] + off);
      }
    }
    F::template cell<LES>(v, K);
    const int po = i + g.sx * j;
    const int o = po + g.sx * g.ny * k;
#pragma unroll
    for (int q = 0; q < Q; ++q) dst.p[q][o] = v[q];
    if (EDGE && k == g.nz - 1) {
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (czq(q) > 0) h.up[zslot(q)][po] = v[q];
    }
    if (EDGE && k == 0) {
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (czq(q) < 0) h.dn[zslot(q)][po] = v[q];
    }
  }
  if (EDGE) {
    // the block's stores into the neighbour's planes (peer memory when the
    // neighbour is another GPU) are made visible system-wide before the
    // kernel ends: a block barrier, then one system-scope fence (cumulative
    // over the stores the barrier ordered before it)
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) __threadfence_system();
  }
}

// Fills the neighbours' ghost planes from this slab's current boundary planes
// (after an initial condition, an upload or a restart).
template <class S>
__global__ void k_halo_prime(Pops<const S> a, Geo g, Halo<S> h) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  if (i < g.nx) {
    const int po = i + g.sx * j;
    const long long top = po + (long long)g.sx * g.ny * (g.nz - 1);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (czq(q) > 0) h.up[zslot(q)][po] = a.p[q][top];
      if (czq(q) < 0) h.dn[zslot(q)][po] = a.p[q][po];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) __threadfence_system();
}

// ------------------------------------------------------------ row units
// Rows of a box as units of 32 cells, one per warp: the decode is two 32-bit
// divisions per warp and unit, and every neighbour offset of a lane is a sum of
// one of three x, row and plane offsets. (With 64-bit divisions and wraps per
// access the diagnostics took 750 us in FP32 and FP16 at 256^3, against 196 and
// 98 us for their bytes at the copy rate: bound by index arithmetic.)
struct Units {
  unsigned per_row, per_plane, n;
  __host__ __device__ explicit Units(int nx, int ny, int nz)
      : per_row((nx + 31) / 32), per_plane(per_row * ny), n(per_plane * nz) {}
  __device__ void decode(unsigned u, int& i, int& j, int& k) const {
    const unsigned z = u / per_plane, r = u - z * per_plane, y = r / per_row;
    k = (int)z;
    j = (int)y;
    i = (int)((r - y * per_row) * 32 + (threadIdx.x & 31));
  }
};

// Offsets of the cells around (i, j, k): off(dx, dy, dz), each -1, 0 or 1.
struct Around {
  int x[3], y[3], z[3];
  __device__ Around(const Geo& g, int i, int j, int k) {
    const int plane = g.sx * g.ny;
    x[0] = i == 0 ? g.nx - 1 : i - 1;
    x[1] = i;
    x[2] = i == g.nx - 1 ? 0 : i + 1;
    y[0] = g.sx * (j == 0 ? g.ny - 1 : j - 1);
    y[1] = g.sx * j;
    y[2] = g.sx * (j == g.ny - 1 ? 0 : j + 1);
    z[0] = plane * (k == 0 ? g.nz - 1 : k - 1);
    z[1] = plane * k;
    z[2] = plane * (k == g.nz - 1 ? 0 : k + 1);
  }
  __device__ int off(int dx, int dy, int dz) const { return x[dx + 1] + y[dy + 1] + z[dz + 1]; }
};

// ------------------------------------------------------ initial conditions
// Per-cell equilibrium deviation of SRC/init.F90:97-137 (cte1 = 0):
// out_q = crho*w_q*(0 + rf*(c.u) + qf*(3*(c.u)^2 - |u|^2)), with each linear
// and quadratic term written as in the reference text.
template <class V>
__device__ __forceinline__ void eq_init(V xj, V yj, V zj, V crho, V (&out)[Q]) {
  using N = Num<V>;
  const V rf = N::c(3.0), qf = N::c(1.5), three = N::c(3.0), zero = N::c(0.0), cte1 = zero;
  const V p0 = N::c(1.0 / 3.0), p1 = N::c(1.0 / 18.0), p2 = N::c(1.0 / (3.0 * 3.0 * (1.0 + 3.0)));
  const V cvsq = xj * xj + yj * yj + zj * zj;
  V cx[Q];
  cx[0]  = rf * (xj - yj) + qf * (three * (xj - yj) * (xj - yj) - cvsq);
  cx[1]  = rf * (xj - zj) + qf * (three * (xj - zj) * (xj - zj) - cvsq);
  cx[2]  = rf * (xj + yj) + qf * (three * (xj + yj) * (xj + yj) - cvsq);
  cx[3]  = rf * (xj + zj) + qf * (three * (xj + zj) * (xj + zj) - cvsq);
  cx[4]  = rf * (xj) + qf * (three * (xj) * (xj) - cvsq);
  cx[5]  = rf * (zj) + qf * (three * (zj) * (zj) - cvsq);
  cx[6]  = rf * (yj + zj) + qf * (three * (yj + zj) * (yj + zj) - cvsq);
  cx[7]  = rf * (yj) + qf * (three * (yj) * (yj) - cvsq);
  cx[8]  = rf * (yj - zj) + qf * (three * (yj - zj) * (yj - zj) - cvsq);
  cx[9]  = rf * (-xj - yj) + qf * (three * (xj + yj) * (xj + yj) - cvsq);
  cx[10] = rf * (-xj - zj) + qf * (three * (xj + zj) * (xj + zj) - cvsq);
  cx[11] = rf * (-xj + yj) + qf * (three * (xj - yj) * (xj - yj) - cvsq);
  cx[12] = rf * (-xj + zj) + qf * (three * (xj - zj) * (xj - zj) - cvsq);
  cx[13] = rf * (-xj) + qf * (three * (xj) * (xj) - cvsq);
  cx[14] = rf * (-zj) + qf * (three * (zj) * (zj) - cvsq);
  cx[15] = rf * (-yj - zj) + qf * (three * (yj + zj) * (yj + zj) - cvsq);
  cx[16] = rf * (-yj) + qf * (three * (yj) * (yj) - cvsq);
  cx[17] = rf * (-yj + zj) + qf * (three * (yj - zj) * (yj - zj) - cvsq);
  cx[18] = rf * zero + qf * (three * zero * zero - cvsq);
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const bool w1 = (q == 4 || q == 5 || q == 7 || q == 13 || q == 14 || q == 16);
    const V w = q == 18 ? p0 : (w1 ? p1 : p2);
    out[q] = crho * w * (cte1 + cx[q]);
  }
}

__device__ __forceinline__ double dsin(double x) { return sin(x); }
__device__ __forceinline__ double dcos(double x) { return cos(x); }
__device__ __forceinline__ float dsin(float x) { return sinf(x); }
__device__ __forceinline__ float dcos(float x) { return cosf(x); }

template <class F>
__device__ __forceinline__ void store_cell(Pops<typename F::S>& a, int lay, int o, typename F::V (&v)[Q],
                                           typename F::R scale) {
  using N = Num<typename F::V>;
#pragma unroll
  for (int q = 0; q < Q; ++q) a.p[lay == LAY_AAE ? oppq(q) : q][o] = F::enc(N::raw(v[q]), scale);
}

// Largest |deviation| of a cell, for choosing the FP16 scale.
template <class V>
__device__ __forceinline__ float cell_maxabs(const V (&v)[Q]) {
  float m = 0.f;
#pragma unroll
  for (int q = 0; q < Q; ++q) m = fmaxf(m, fabsf((float)Num<V>::raw(v[q])));
  return m;
}

// Taylor-Green vortex, SRC/init.F90:83-141 (offsets zero, one box).
// maxbits != nullptr: measure max |deviation| only (atomicMax on the bits of a
// non-negative float), store nothing.
template <class F>
__global__ void k_init_tgv(Pops<typename F::S> a, Geo g, int lay, typename F::R u0r, int faithful,
                           typename F::R scale, unsigned int* maxbits) {
  using R = typename F::R; using V = typename F::V; using N = Num<V>;
  const long long n = (long long)g.nx * g.ny * g.nz;
  float tmax = 0.f;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(c % g.nx), j = (int)((c / g.nx) % g.ny), k = (int)(c / ((long long)g.nx * g.ny));
    // reference interior indices are 1-based; a z-slab uses global z
    // (k0 + k with k0 = offset(3), SRC/init.F90:73,84)
    const int ir = i + 1, jr = j + 1, kr = g.z0 + k + 1;
    const int gz = g.gz > 0 ? g.gz : g.nz;
    R x, y, z, pi;
    if (faithful) {
      x = (R)(((float)ir - 0.5f) / (float)g.nx);
      y = (R)(((float)jr - 0.5f) / (float)g.ny);
      z = (R)(((float)kr - 0.5f) / (float)gz);
      pi = (R)3.141592653589793238462643383279f;
    } else {
      x = (R)(((double)ir - 0.5) / (double)g.nx);
      y = (R)(((double)jr - 0.5) / (double)g.ny);
      z = (R)(((double)kr - 0.5) / (double)gz);
      pi = (R)3.141592653589793238462643383279;
    }
    const V two = N::c(2.0), four = N::c(4.0), u0 = N::wrap(u0r), P = N::wrap(pi);
    const V X = N::wrap(x), Y = N::wrap(y), Z = N::wrap(z);
    const R ax = N::raw(two * P * X), ay = N::raw(two * P * Y), az = N::raw(two * P * Z);
    const V xj = u0 * N::wrap(dsin(ax)) * N::wrap(dcos(ay)) * N::wrap(dcos(az));
    const V yj = -(u0 * N::wrap(dcos(ax)) * N::wrap(dsin(ay)) * N::wrap(dcos(az)));
    const V zj = N::c(0.0);
    V crho = N::c(1.0);
    if (faithful) {
      const R bx = N::raw(four * P * X), by = N::raw(four * P * Y), bz = N::raw(four * P * Z);
      crho = N::c(1.0) + ((u0 * u0) / (N::c(16.0) * N::c(3.0))) * (N::wrap(dcos(bx)) + N::wrap(dcos(by))) *
                             (N::wrap(dcos(bz)) + N::c(2.0));
    }
    V out[Q];
    eq_init<V>(xj, yj, zj, crho, out);
    if (maxbits) tmax = fmaxf(tmax, cell_maxabs<V>(out));
    else store_cell<F>(a, lay, i + g.sx * (j + g.ny * k), out, scale);
  }
  if (maxbits) atomicMax(maxbits, __float_as_uint(tmax));
}

// Equilibrium from a staged velocity slab (planes k0 .. k0+nk-1, dense
// Fortran order) at uniform density rho.
template <class F>
__global__ void k_init_vel(Pops<typename F::S> a, Geo g, int lay, const double* __restrict__ u,
                           const double* __restrict__ v, const double* __restrict__ w, double rho, int k0, int nk,
                           typename F::R scale, unsigned int* maxbits) {
  using R = typename F::R; using V = typename F::V; using N = Num<V>;
  float tmax = 0.f;
  const Units un(g.nx, g.ny, nk);
  for (unsigned m = blockIdx.x * 8 + (threadIdx.x >> 5); m < un.n; m += gridDim.x * 8) {
    int i, j, k;
    un.decode(m, i, j, k);
    if (i >= g.nx) continue;
    const long long c = i + (long long)g.nx * (j + (long long)g.ny * k);
    V out[Q];
    eq_init<V>(N::wrap((R)u[c]), N::wrap((R)v[c]), N::wrap((R)w[c]), N::wrap((R)rho), out);
    if (maxbits) tmax = fmaxf(tmax, cell_maxabs<V>(out));
    else store_cell<F>(a, lay, i + g.sx * (j + g.ny * (k0 + k)), out, scale);
  }
  if (maxbits) atomicMax(maxbits, __float_as_uint(tmax));
}

// ------------------------------------------------------- reference access
// Location of the reference's a_q at cell (i,j,k) + d for a given layout.
template <int LAY>
__device__ __forceinline__ int ref_slot(int q) { return LAY == LAY_AAE ? oppq(q) : q; }
// Location of the reference's a_q of the cell (local) and of its pulled a_q,
// from (x - c_q), for a layout: LAY_AAN keeps a_q of a cell at x + c_q.
template <int LAY, bool PULL>
__device__ __forceinline__ int around_off(const Around& n, int q) {
  constexpr int s = PULL ? (LAY == LAY_AAN ? 0 : -1) : (LAY == LAY_AAN ? 1 : 0);
  return n.off(s * cxq(q), s * cyq(q), s * czq(q));
}

// Populations q0 .. q0 + nq - 1 of the reference to nq dense blocks: stored type
// (out_s) or double deviations (out_d).
template <class F, int LAY>
__global__ void __launch_bounds__(256) k_export(Pops<const typename F::S> a, Geo g, int q0, int nq,
                                                typename F::S* out_s, double* out_d, typename F::R inv) {
  const long long n = (long long)g.nx * g.ny * g.nz;
  const Units un(g.nx, g.ny, g.nz);
  for (unsigned u = blockIdx.x * 8 + (threadIdx.x >> 5); u < un.n; u += gridDim.x * 8) {
    int i, j, k;
    un.decode(u, i, j, k);
    if (i >= g.nx) continue;
    const Around nb(g, i, j, k);
    const long long c = i + (long long)g.nx * (j + (long long)g.ny * k);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (q < q0 || q >= q0 + nq) continue;
      const typename F::S s = ldg(a.p[ref_slot<LAY>(q)] + around_off<LAY, false>(nb, q));
      if (out_s) out_s[(q - q0) * n + c] = s;
      if (out_d) out_d[(q - q0) * n + c] = (double)F::dec(s, inv);
    }
  }
}

// The inverse of k_export's stored form.
template <class F, int LAY>
__global__ void __launch_bounds__(256) k_import(Pops<typename F::S> a, Geo g, int q0, int nq,
                                                const typename F::S* __restrict__ in) {
  const long long n = (long long)g.nx * g.ny * g.nz;
  const Units un(g.nx, g.ny, g.nz);
  for (unsigned u = blockIdx.x * 8 + (threadIdx.x >> 5); u < un.n; u += gridDim.x * 8) {
    int i, j, k;
    un.decode(u, i, j, k);
    if (i >= g.nx) continue;
    const Around nb(g, i, j, k);
    const long long c = i + (long long)g.nx * (j + (long long)g.ny * k);
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (q >= q0 && q < q0 + nq) a.p[ref_slot<LAY>(q)][around_off<LAY, false>(nb, q)] = in[(q - q0) * n + c];
  }
}

// ------------------------------------------------------------ diagnostics
// Quantities: 0 rho, 1 ux, 2 uy, 3 uz, 4 0.5|u|^2 (local populations,
// SRC/diagno.F90:96-111); 5 0.5|u|^2, 6 2*svisc*Ptotal (pulled populations,
// SRC/dissipation.F90:76-249); 7 2*nu*S:S with S = -3*omega*Pi/(2*rho);
// 8 non-finite cell count; 9 enstrophy (k_enstrophy).
// Offset of the periodic image of an out-of-box source cell (si, sj, sk) in a
// population's block of a boundary-plane snapshot: x planes (ny*nz each), then
// y planes (nx*nz), then z planes (nx*ny).
__device__ __forceinline__ long long faith_off(const Geo& g, int si, int sj, int sk) {
  const int wi = wrapi(si, g.nx), wj = wrapi(sj, g.ny), wk = wrapi(sk, g.nz);
  const long long yz = (long long)g.ny * g.nz, xz = (long long)g.nx * g.nz, xy = (long long)g.nx * g.ny;
  if (si < 0 || si >= g.nx) return (wi == 0 ? 0 : yz) + wj + (long long)g.ny * wk;
  if (sj < 0 || sj >= g.ny) return 2 * yz + (wj == 0 ? 0 : xz) + wi + (long long)g.nx * wk;
  return 2 * (yz + xz) + (wk == 0 ? 0 : xy) + wi + (long long)g.nx * wj;
}

template <class S>
__global__ void k_faith_snapshot(Pops<const S> a, Geo g, S* out) {
  const long long yz = (long long)g.ny * g.nz, xz = (long long)g.nx * g.nz, xy = (long long)g.nx * g.ny;
  const long long per = 2 * (yz + xz + xy), n = (long long)Q * per;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
    const int q = (int)(e / per);
    long long r = e % per;
    int i, j, k;
    if (r < 2 * yz) {
      i = r < yz ? 0 : g.nx - 1;
      r %= yz;
      j = (int)(r % g.ny);
      k = (int)(r / g.ny);
    } else if (r < 2 * (yz + xz)) {
      r -= 2 * yz;
      j = r < xz ? 0 : g.ny - 1;
      r %= xz;
      i = (int)(r % g.nx);
      k = (int)(r / g.nx);
    } else {
      r -= 2 * (yz + xz);
      k = r < xy ? 0 : g.nz - 1;
      r %= xy;
      i = (int)(r % g.nx);
      j = (int)(r / g.nx);
    }
    out[e] = a.p[q][i + (long long)g.sx * (j + (long long)g.ny * k)];
  }
}

// Sources of the pulls that leave the box or the slab: the periodic image
// (PULL_WRAP), the ghost planes of a z-slab (PULL_SLAB), the boundary-plane
// snapshot of faithful mode (PULL_FAITH).
enum { PULL_WRAP = 0, PULL_SLAB = 1, PULL_FAITH = 2 };
constexpr int NDK = 9;  // quantities of k_diag

// Blocks of k_diag: what the SMs hold at once (128 registers in FP64, 80 in the
// others), so that no second wave runs half empty. 256^3, us, with 592 blocks and
// so: FP64 727 / 659, FP32 644 / 510, FP16 602 / 513.
__host__ __device__ constexpr int diag_blocks_per_sm(int form) { return form == FORM_F64 ? 2 : 3; }
static int diag_blocks(int form) { return 148 * diag_blocks_per_sm(form); }

template <class F, int LAY, int PULL>
__global__ void __launch_bounds__(DIAG_THREADS, diag_blocks_per_sm(F::id))
    k_diag(Pops<const typename F::S> a, Geo g, double svisc, double omega, typename F::R inv, double* partials,
           typename F::R* vel, Halo<typename F::S> h, const typename F::S* faith, int faith_zero) {
  step_begin();
  using R = typename F::R; using V = typename F::V; using N = Num<V>;
  __shared__ KS sh[DIAG_THREADS / 32][NDK];
  KS acc[NDK];
#pragma unroll
  for (int d = 0; d < NDK; ++d) acc[d] = {0.0, 0.0};
  int bad = 0;
  const long long n = (long long)g.nx * g.ny * g.nz;
  const V svr = N::wrap((R)svisc);
  const double kS = 2.0 * svisc * (9.0 * omega * omega * 0.25);  // 2 nu S:S = kS Ptotal / rho^2
  const Units un(g.nx, g.ny, g.nz);
  constexpr unsigned WARPS = DIAG_THREADS / 32;
  for (unsigned u = blockIdx.x * WARPS + (threadIdx.x >> 5); u < un.n; u += gridDim.x * WARPS) {
    int i, j, k;
    un.decode(u, i, j, k);
    if (i >= g.nx) continue;
    const Around nb(g, i, j, k);
    V x[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q)
      x[q] = N::wrap(F::dec(a.p[ref_slot<LAY>(q)][around_off<LAY, false>(nb, q)], inv));
    V ux, uy, uz;
    const V rho = moments<V>(x, ux, uy, uz);
    const V ke = N::c(0.5) * (ux * ux + uy * uy + uz * uz);
    kadd(acc[0], (double)N::raw(rho));
    kadd(acc[1], (double)N::raw(ux));
    kadd(acc[2], (double)N::raw(uy));
    kadd(acc[3], (double)N::raw(uz));
    kadd(acc[4], (double)N::raw(ke));
    if (!isfinite(N::raw(rho)) || !isfinite(N::raw(ux)) || !isfinite(N::raw(uy)) || !isfinite(N::raw(uz))) ++bad;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int si = i - cxq(q), sj = j - cyq(q), sk = k - czq(q);
      if (PULL == PULL_SLAB && ((czq(q) > 0 && k == 0) || (czq(q) < 0 && k == g.nz - 1))) {
        // a z-slab pulls across its faces from its ghost planes
        const int po = nb.off(-cxq(q), -cyq(q), 0) - nb.z[1];
        x[q] = N::wrap(F::dec(czq(q) > 0 ? h.in_lo[zslot(q)][po] : h.in_hi[zslot(q)][po], inv));
      } else if (PULL == PULL_FAITH && (si < 0 || si >= g.nx || sj < 0 || sj >= g.ny || sk < 0 || sk >= g.nz)) {
        // faithful mode: the reference's ghost cell of this pull, filled two
        // steps earlier (or never)
        const long long per = 2 * ((long long)g.ny * g.nz + (long long)g.nx * g.nz + (long long)g.nx * g.ny);
        x[q] = faith_zero ? N::c(0.0) : N::wrap(F::dec(faith[q * per + faith_off(g, si, sj, sk)], inv));
      } else {
        x[q] = N::wrap(F::dec(a.p[ref_slot<LAY>(q)][around_off<LAY, true>(nb, q)], inv));
      }
    }
    if (vel) {  // behind the pulls: none of these loads may move over a store
      const long long c = i + (long long)g.nx * (j + (long long)g.ny * k);
      vel[c] = N::raw(ux);
      vel[n + c] = N::raw(uy);
      vel[2 * n + c] = N::raw(uz);
    }
    V e[Q], vx, vy, vz;
    const V rp = equilibrium<V>(x, e, vx, vy, vz);
    const V vsq = vx * vx + vy * vy + vz * vz;
    const V P = ptotal<V>(x, e);
    kadd(acc[5], (double)N::raw(N::c(0.5) * vsq));
    kadd(acc[6], (double)N::raw(N::c(2.0) * svr * P));
    const double r = __drcp_rn((double)N::raw(rp));
    kadd(acc[7], __dmul_rn(__dmul_rn(kS, __dmul_rn(r, r)), (double)N::raw(P)));
  }
  acc[8].s = (double)bad;
  const KS r = block_reduce_n<NDK, DIAG_THREADS>(acc, sh);
  constexpr int W = DIAG_THREADS / 32;
  if (threadIdx.x % W == 0 && threadIdx.x / W < NDK) {
    partials[(blockIdx.x * ND + threadIdx.x / W) * 2 + 0] = r.s;
    partials[(blockIdx.x * ND + threadIdx.x / W) * 2 + 1] = r.c;
  }
}

// Local velocity j/rho of the cells of planes k0 .. k0 + nk - 1, dense Fortran
// order (three blocks), in OUT precision: what k_diag also writes, for callers that want nothing else
// (bgk_get_velocity, bgk_spectrum). 19 loads and 3 stores a cell.
template <class F, int LAY, class OUT>
__global__ void __launch_bounds__(256) k_velocity(Pops<const typename F::S> a, Geo g, typename F::R inv, OUT* vel,
                                                  int k0, int nk) {
  using V = typename F::V; using N = Num<V>;
  const long long n = (long long)g.nx * g.ny * nk;
  const Units un(g.nx, g.ny, nk);
  for (unsigned u = blockIdx.x * 8 + (threadIdx.x >> 5); u < un.n; u += gridDim.x * 8) {
    int i, j, k;
    un.decode(u, i, j, k);
    if (i >= g.nx) continue;
    const Around nb(g, i, j, k0 + k);
    V x[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q)
      x[q] = N::wrap(F::dec(ldg(a.p[ref_slot<LAY>(q)] + around_off<LAY, false>(nb, q)), inv));
    V ux, uy, uz;
    (void)moments<V>(x, ux, uy, uz);
    const long long c = i + (long long)g.nx * (j + (long long)g.ny * k);
    vel[c] = (OUT)N::raw(ux);
    vel[n + c] = (OUT)N::raw(uy);
    vel[2 * n + c] = (OUT)N::raw(uz);
  }
}

template <class R>
__global__ void __launch_bounds__(DIAG_THREADS) k_enstrophy(const R* vel, int nx, int ny, int nz,
                                                           double* partials) {
  step_begin();
  __shared__ KS sh[DIAG_THREADS / 32][1];
  KS acc[1] = {{0.0, 0.0}};
  const long long n = (long long)nx * ny * nz;
  const Units un(nx, ny, nz);
  constexpr unsigned WARPS = DIAG_THREADS / 32;
  for (unsigned u = blockIdx.x * WARPS + (threadIdx.x >> 5); u < un.n; u += gridDim.x * WARPS) {
    int i, j, k;
    un.decode(u, i, j, k);
    if (i >= nx) continue;
    const int ip = i + 1 == nx ? 0 : i + 1, im = i == 0 ? nx - 1 : i - 1;
    const int jp = j + 1 == ny ? 0 : j + 1, jm = j == 0 ? ny - 1 : j - 1;
    const int kp = k + 1 == nz ? 0 : k + 1, km = k == 0 ? nz - 1 : k - 1;
    // rows of the three components at (j, k) and around it
    const R* const row = vel + (long long)nx * (j + (long long)ny * k);
    const R* const rjp = vel + (long long)nx * (jp + (long long)ny * k);
    const R* const rjm = vel + (long long)nx * (jm + (long long)ny * k);
    const R* const rkp = vel + (long long)nx * (j + (long long)ny * kp);
    const R* const rkm = vel + (long long)nx * (j + (long long)ny * km);
    using E = Ex<double>;
    auto D = [&](const R* p, int s, const R* m, int t) -> E { return E{0.5} * (E{(double)p[s]} - E{(double)m[t]}); };
    const E dwdy = D(rjp + 2 * n, i, rjm + 2 * n, i), dvdz = D(rkp + n, i, rkm + n, i);
    const E dudz = D(rkp, i, rkm, i), dwdx = D(row + 2 * n, ip, row + 2 * n, im);
    const E dvdx = D(row + n, ip, row + n, im), dudy = D(rjp, i, rjm, i);
    const E wx = dwdy - dvdz, wy = dudz - dwdx, wz = dvdx - dudy;
    kadd(acc[0], (E{0.5} * (wx * wx + wy * wy + wz * wz)).v);
  }
  const KS r = block_reduce_n<1, DIAG_THREADS>(acc, sh);
  if (threadIdx.x == 0) {
    partials[(blockIdx.x * ND + 9) * 2 + 0] = r.s;
    partials[(blockIdx.x * ND + 9) * 2 + 1] = r.c;
  }
}

// One block per quantity (one block for all ten took 16 us). totals may be
// pinned host memory; err (optional): the device's error flag, copied behind
// the ND + 1 totals so that the host reads one place.
__global__ void __launch_bounds__(DIAG_THREADS) k_finalize(const double* partials, int blocks,
                                                           double* totals, const int* err) {
  step_begin();
  __shared__ KS sh[DIAG_THREADS / 32][1];
  const int d = blockIdx.x;
  KS acc[1] = {{0.0, 0.0}};
  const int nb = d < NDK ? blocks : DIAG_BLOCKS;  // k_diag's, k_enstrophy's
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    const double2 p = reinterpret_cast<const double2*>(partials)[b * ND + d];
    kcomb(acc[0], KS{p.x, p.y});
  }
  const KS r = block_reduce_n<1, DIAG_THREADS>(acc, sh);
  if (threadIdx.x == 0) {
    totals[d] = __dadd_rn(r.s, r.c);
    if (d == 0 && err) totals[ND + 1] = (double)*err;
  }
}

template <class F, int LAY>
__global__ void k_last_zj(Pops<const typename F::S> a, Geo g, typename F::R inv, double* out) {
  using V = typename F::V; using N = Num<V>;
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const Around nb(g, g.nx - 1, g.ny - 1, g.nz - 1);
  V x[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q)
    x[q] = N::wrap(F::dec(a.p[ref_slot<LAY>(q)][around_off<LAY, false>(nb, q)], inv));
  V ux, uy, uz;
  (void)moments<V>(x, ux, uy, uz);
  *out = (double)N::raw(uz);
}

// -------------------------------------------------------------------- VTK
// Velocity j/rho of the points of a VTK slice or box, as float triples in the
// file order of SRC/vtk_xy.binary.F90:79-97 (xy: j outer, i inner), vtk_xz
// (k, i), vtk_yz (k, j) and vtk_3d (k, j, i). The sums are taken in the
// storage arithmetic in the reference's order, each rounded to single
// precision, then divided in single precision (u/den).
template <class F, int LAY>
__global__ void k_vtk(Pops<const typename F::S> a, Geo g, int kind, int index, float* out, long long npts,
                      typename F::R inv) {
  using V = typename F::V; using N = Num<V>;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < npts; c += (long long)gridDim.x * blockDim.x) {
    int i, j, k;
    if (kind == 1) { i = (int)(c % g.nx); j = (int)(c / g.nx); k = index; }
    else if (kind == 2) { i = (int)(c % g.nx); k = (int)(c / g.nx); j = index; }
    else if (kind == 3) { j = (int)(c % g.ny); k = (int)(c / g.ny); i = index; }
    else { i = (int)(c % g.nx); j = (int)((c / g.nx) % g.ny); k = (int)(c / ((long long)g.nx * g.ny)); }
    const Around nb(g, i, j, k);
    V x[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) x[q] = N::wrap(F::dec(a.p[ref_slot<LAY>(q)][around_off<LAY, false>(nb, q)], inv));
    const V u = x[0] + x[1] + x[2] + x[3] + x[4] - x[9] - x[10] - x[11] - x[12] - x[13];
    const V w = x[2] + x[6] + x[7] + x[8] + x[11] - x[0] - x[9] - x[15] - x[16] - x[17];
    const V v = x[3] + x[5] + x[6] + x[12] + x[17] - x[1] - x[8] - x[10] - x[14] - x[15];
    const V den = x[0] + x[1] + x[2] + x[3] + x[4] + x[5] + x[6] + x[7] + x[8] + x[9] + x[10] + x[11] + x[12] +
                  x[13] + x[14] + x[15] + x[16] + x[17] + x[18] + N::c(1.0);
    const float d = (float)N::raw(den);
    out[3 * c + 0] = __fdiv_rn((float)N::raw(u), d);
    out[3 * c + 1] = __fdiv_rn((float)N::raw(w), d);
    out[3 * c + 2] = __fdiv_rn((float)N::raw(v), d);
  }
}

// --------------------------------------------------------------- spectrum
// Shell of a wavevector: floor(|k| + 1/2), in integers (b^2 - b < |k|^2 <= b^2 + b).
__device__ __forceinline__ int shell_of(int k2) {
  int b = (int)(__fsqrt_rn((float)k2) + 0.5f);
  if (k2 > b * b + b) ++b;
  else if (b > 0 && k2 <= b * b - b) --b;
  return b;
}

constexpr int SPEC_WARPS = 8;
constexpr int SPEC_MAX_SIDE = 16384;  // |k|^2 and b^2 + b stay below 2^31

// One transformed component into the shells. A warp takes 32 consecutive modes
// of a row, whose shells never decrease from lane to lane (kx >= 0): a segmented
// sum over the lanes leaves one value per shell, added without atomics to the
// warp's own table in shared memory; the block adds its tables to the result
// at the end. (A global atomic per mode took 1060 us per component at 256^3
// FP64, against 21 us for reading it at the copy rate.)
template <class C>
__global__ void __launch_bounds__(32 * SPEC_WARPS) k_spec_bins(const C* __restrict__ f, int nx, int ny, int nz,
                                                               int nb, double* bins, double norm) {
  extern __shared__ double tab[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int b = threadIdx.x; b < SPEC_WARPS * nb; b += blockDim.x) tab[b] = 0.0;
  __syncthreads();
  double* const own = tab + w * nb;
  const int nxh = nx / 2 + 1;
  const Units un(nxh, ny, nz);
  for (unsigned u = blockIdx.x * SPEC_WARPS + w; u < un.n; u += gridDim.x * SPEC_WARPS) {
    int ix, iy, iz;
    un.decode(u, ix, iy, iz);
    const int ky = iy <= ny / 2 ? iy : iy - ny, kz = iz <= nz / 2 ? iz : iz - nz;
    double v = 0.0;
    int b = nb;
    if (ix < nxh) {
      const C c = f[ix + (long long)nxh * (iy + (long long)ny * iz)];
      // modes 0 < kx < nx/2 stand for their conjugate partner as well
      const double wt = (ix == 0 || (nx % 2 == 0 && ix == nx / 2)) ? 1.0 : 2.0;
      const double re = (double)c.x, im = (double)c.y;
      v = wt * 0.5 * (re * re + im * im) * norm;
      b = min(nb, shell_of(ix * ix + ky * ky + kz * kz));
    }
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const double o = __shfl_up_sync(0xffffffffu, v, s);
      const int ob = __shfl_up_sync(0xffffffffu, b, s);
      if (lane >= s && ob == b) v += o;
    }
    const int next = __shfl_down_sync(0xffffffffu, b, 1);
    if (b < nb && (lane == 31 || next != b)) own[b] += v;
    __syncwarp();
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    double v = 0.0;
    for (int m = 0; m < SPEC_WARPS; ++m) v += tab[m * nb + b];
    if (v != 0.0) atomicAdd(bins + b, v);
  }
}

// The same for boxes whose shells do not fit the tables: one atomic per mode.
template <class C>
__global__ void k_spec_bins_any(const C* __restrict__ f, int nx, int ny, int nz, int nbins, double* bins, double norm) {
  const int nxh = nx / 2 + 1;
  const long long n = (long long)nxh * ny * nz;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    const int ix = (int)(c % nxh), iy = (int)((c / nxh) % ny), iz = (int)(c / ((long long)nxh * ny));
    const int ky = iy <= ny / 2 ? iy : iy - ny, kz = iz <= nz / 2 ? iz : iz - nz;
    const double w = (ix == 0 || (nx % 2 == 0 && ix == nx / 2)) ? 1.0 : 2.0;
    const double kk = sqrt((double)ix * ix + (double)ky * ky + (double)kz * kz);
    const int b = (int)floor(kk + 0.5);
    if (b < nbins) {
      const double re = (double)f[c].x, im = (double)f[c].y;
      atomicAdd(bins + b, w * 0.5 * (re * re + im * im) * norm);
    }
  }
}

template <class C>
static cudaError_t spec_impl(const void* fft_out, int nx, int ny, int nz, int nbins, double* bins, double norm,
                             cudaStream_t st) {
  const double kmax = std::sqrt(0.25 * ((double)nx * nx + (double)ny * ny + (double)nz * nz));
  const int nb = (int)std::min((double)nbins, std::floor(kmax + 0.5) + 1.0);  // shells above hold nothing
  const size_t bytes = (size_t)SPEC_WARPS * nb * sizeof(double);
  if (nx <= SPEC_MAX_SIDE && ny <= SPEC_MAX_SIDE && nz <= SPEC_MAX_SIDE && bytes <= 48 * 1024) {
    const int grid = grid_1d(Units(nx / 2 + 1, ny, nz).n, SPEC_WARPS, 148 * 4);
    k_spec_bins<C><<<grid, 32 * SPEC_WARPS, bytes, st>>>((const C*)fft_out, nx, ny, nz, nb, bins, norm);
  } else {
    const long long n = (long long)(nx / 2 + 1) * ny * nz;
    k_spec_bins_any<C><<<grid_1d(n, 256, 148 * 16), 256, 0, st>>>((const C*)fft_out, nx, ny, nz, nbins, bins, norm);
  }
  return cudaGetLastError();
}

cudaError_t launch_spectrum_bins(const void* fft_out, int form, int nx, int ny, int nz, int nbins, double* bins,
                                 double norm, cudaStream_t st) {
  return form == FORM_F64 ? spec_impl<double2>(fft_out, nx, ny, nz, nbins, bins, norm, st)
                          : spec_impl<float2>(fft_out, nx, ny, nz, nbins, bins, norm, st);
}

// ---------------------------------------------------------------- shift3
template <class T>
__global__ void k_shift3(const T* __restrict__ i1, const T* __restrict__ i2, const T* __restrict__ i3, T* o1, T* o2,
                         T* o3, int nx, int ny, int nz, int dir) {
  const long long n = (long long)nx * ny * nz;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(c % nx), j = (int)((c / nx) % ny), k = (int)(c / ((long long)nx * ny));
    const long long rowj = (long long)nx * (j + (long long)ny * k);
    const int is = wrapi(i - dir, nx), js = wrapi(j - dir, ny), ks = wrapi(k - dir, nz);
    o1[c] = __ldg(i1 + rowj + is);
    o2[c] = __ldg(i2 + i + (long long)nx * (js + (long long)ny * k));
    o3[c] = __ldg(i3 + i + (long long)nx * (j + (long long)ny * ks));
  }
}

// ============================================================== launchers
template <class S> static Pops<S> pops_of(const Lattice& L) {
  Pops<S> p;
  for (int q = 0; q < Q; ++q) p.p[q] = (S*)L.p[q];
  return p;
}

StepK make_stepk(int form, double omega, double scale, double les_cs) {
  StepK k{};
  k.omega = omega;
  k.omega_f = (float)omega;
  k.inv = (float)(1.0 / scale);
  k.om1 = 1.0f - (float)omega;
  k.scale = (float)scale;
  const double w[3] = {1.0 / 3.0, 1.0 / 18.0, 1.0 / 36.0};
  for (int c = 0; c < 3; ++c) k.kw[c] = (float)((double)(float)omega * scale * w[c]);
  // Smagorinsky constants of SRC/col_MC.F90:305 in the form's arithmetic:
  // 18*(cteS)**2, 1/(2*omega1) and (1/omega1)**2 (host code is built without
  // contraction, so each operation rounds as written)
  k.les = les_cs > 0.0;
  if (k.les) {
    k.cs18 = 18.0 * (les_cs * les_cs);
    k.tauh = 1.0 / (2.0 * omega);
    k.tau2 = (1.0 / omega) * (1.0 / omega);
    const float cs = (float)les_cs, om = (float)omega;
    k.cs18_f = 18.0f * (cs * cs);
    k.tauh_f = 1.0f / (2.0f * om);
    k.tau2_f = (1.0f / om) * (1.0f / om);
  }
  (void)form;
  return k;
}

// Launches a several-cells-per-thread kernel (its aligned and its flat
// instantiation) in 128-thread blocks over the threads of `planes` planes.
template <class... P, class... A>
static cudaError_t launch_vec(void (*aligned)(P...), void (*flat)(P...), const Geo& g, const VecRows& r, int planes,
                              cudaStream_t st, A... args) {
  const dim3 grid((unsigned)(((long long)g.ny * r.tpr + 127) / 128), (unsigned)planes);
  return launch_step(r.flat ? flat : aligned, grid, dim3(128), st, args...);
}
// The same as an ordinary launch, for a stream that is ordered by events.
template <class... P, class... A>
static void launch_vec_plain(void (*aligned)(P...), void (*flat)(P...), const Geo& g, const VecRows& r, int planes,
                             cudaStream_t st, A... args) {
  const dim3 grid((unsigned)(((long long)g.ny * r.tpr + 127) / 128), (unsigned)planes);
  if (r.flat) flat<<<grid, 128, 0, st>>>(P(args)...);
  else aligned<<<grid, 128, 0, st>>>(P(args)...);
}

template <class F>
static cudaError_t two_impl(const Lattice& s, const Lattice& d, const StepK& K, int variant, cudaStream_t st) {
  using S = typename F::S;
  Pops<const S> ps = pops_of<const S>(s);
  Pops<S> pd = pops_of<S>(d);
  pd.p[Q - 1] = (S*)s.p[Q - 1];  // pop 19 in place (SRC/col_MC.F90:351)
  Shape sh = cell_shape(s.g);
  const long long cells = (long long)s.g.nx * s.g.ny * s.g.nz;
  // FP32: two cells per thread (automatic or 2): on B200 at 256^3, 43.7 GLUPS
  // against 42.0 with one cell per thread, the Smagorinsky step 43.5 against
  // 40.7; rows of no power of two: 180^3 39.0 against 34.4
  const bool big = cells >= VEC_MIN_TWO;
  if (F::id == FORM_F32 && (variant == 2 || (variant == 0 && big))) {
    Pops<float> pf = pops_of<float>(d);
    pf.p[Q - 1] = (float*)s.p[Q - 1];
    const VecRows r(s.g, 2, true);
    if (K.les) return launch_vec(k_two_f32v<true, false>, k_two_f32v<true, true>, s.g, r, s.g.nz, st, pops_of<const float>(s), pf, s.g, K, r.arg, 0);
    return launch_vec(k_two_f32v<false, false>, k_two_f32v<false, true>, s.g, r, s.g.nz, st, pops_of<const float>(s), pf, s.g, K, r.arg, 0);
  }
  // FP16: four cells per thread (automatic or 4; the Smagorinsky step too), the
  // fastest measured on B200 at 256^3 (76.6 GLUPS against 64.0 with one, 62.7
  // with two and 44.6 for the row pipeline); rows of no power of two: 201 x 163 x 117 71.9
  // against 49.8, 180^3 74.3 against 51.3
  if (F::id == FORM_F16 && (variant == 4 || (variant == 0 && big))) {
    Pops<__half> ph = pops_of<__half>(d);
    ph.p[Q - 1] = (__half*)s.p[Q - 1];
    const VecRows r(s.g, 4, true);
    if (K.les) return launch_vec(k_two_f16v<true, false>, k_two_f16v<true, true>, s.g, r, s.g.nz, st, pops_of<const __half>(s), ph, s.g, K, r.arg, 0);
    return launch_vec(k_two_f16v<false, false>, k_two_f16v<false, true>, s.g, r, s.g.nz, st, pops_of<const __half>(s), ph, s.g, K, r.arg, 0);
  }
  if (K.les) {  // the other choices run the Smagorinsky collision on one cell per thread
    return launch_step(k_two<F, true>, sh.grid, sh.block, st, ps, pd, s.g, K);
  }
  if (variant == 8) {
    bool launched = false;
    cudaError_t e = launch_rows(s, d, ROW_TWO, K, st, &launched);
    if (e != cudaSuccess || launched) return e;
  }
  if (F::id == FORM_F16 && variant == 2) {
    const VecRows r(s.g, 2, true);
    if (!r.flat) {
      Pops<__half> ph = pops_of<__half>(d);
      ph.p[Q - 1] = (__half*)s.p[Q - 1];
      const dim3 grid((unsigned)(((long long)s.g.ny * r.tpr + 255) / 256), s.g.nz);
      return launch_step(k_two_f16v2, grid, 256, st, pops_of<const __half>(s), ph, s.g, K, r.arg);
    }
  }
  return launch_step(k_two<F>, sh.grid, sh.block, st, ps, pd, s.g, K);
}

cudaError_t launch_step_out_of_place(const Lattice& src, const Lattice& dst, double omega, cudaStream_t st) {
  const StepK K = make_stepk(src.form, omega, 1.0);
  const Shape sh = cell_shape(src.g);
  switch (src.form) {
    case FORM_F64:
      return launch_step(k_two<F64>, sh.grid, sh.block, st, pops_of<const double>(src), pops_of<double>(dst), src.g, K);
    case FORM_F32: {
      const VecRows r(src.g, 2, true);
      if (!r.pays(src.g, src.g.nz))
        return launch_step(k_two<F32>, sh.grid, sh.block, st, pops_of<const float>(src), pops_of<float>(dst), src.g, K);
      return launch_vec(k_two_f32v<false, false>, k_two_f32v<false, true>, src.g, r, src.g.nz, st, pops_of<const float>(src),
                 pops_of<float>(dst), src.g, K, r.arg, 0);
    }
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_two_lattice(const Lattice& src, const Lattice& dst, double omega, double scale, double les_cs,
                               int variant, cudaStream_t st) {
  const StepK K = make_stepk(src.form, omega, scale, les_cs);
  switch (src.form) {
    case FORM_F64: return two_impl<F64>(src, dst, K, variant, st);
    case FORM_F32: return two_impl<F32>(src, dst, K, variant, st);
    case FORM_F16: return two_impl<F16>(src, dst, K, variant, st);
  }
  return cudaErrorInvalidValue;
}

template <class F>
static cudaError_t aa_impl(const Lattice& a, int odd, const StepK& K, int variant, cudaStream_t st) {
  using S = typename F::S;
  Shape sh = cell_shape(a.g);
  // FP32 (automatic or 2): two cells per thread; the pair of AA steps measured
  // 41.9 GLUPS against 39.8 with one cell per thread at 256^3 on B200 (40.5
  // against 38.9 at 1024^3), the Smagorinsky pair 40.6 against 34.1. The
  // automatic odd step has four cells per thread where rows are whole chunks:
  // 44.1 GLUPS for the pair at 256^3 and 44.2 at 512^3 against 42.2 and 40.8,
  // with the Smagorinsky collision 43.9 against 40.9
  const bool big = (long long)a.g.nx * a.g.ny * a.g.nz >= VEC_MIN_AA;
  if (F::id == FORM_F32 && (variant == 2 || (variant == 0 && big))) {
    const Pops<float> pf = pops_of<float>(a);
    const VecRows r4(a.g, 4, false, true), r(a.g, 2, false);
    if (odd && variant == 0 && r4.arg >= 0) {
      if (K.les) return launch_vec(k_aa_f32w<true, false>, k_aa_f32w<true, true>, a.g, r4, a.g.nz, st, pf, a.g, K, r4.arg);
      else return launch_vec(k_aa_f32w<false, false>, k_aa_f32w<false, true>, a.g, r4, a.g.nz, st, pf, a.g, K, r4.arg);
    } else if (K.les) {
      if (odd) return launch_vec(k_aa_f32v<true, true, false>, k_aa_f32v<true, true, true>, a.g, r, a.g.nz, st, pf, a.g, K, r.arg);
      else return launch_vec(k_aa_f32v<false, true, false>, k_aa_f32v<false, true, true>, a.g, r, a.g.nz, st, pf, a.g, K, r.arg);
    } else {
      if (odd) return launch_vec(k_aa_f32v<true, false, false>, k_aa_f32v<true, false, true>, a.g, r, a.g.nz, st, pf, a.g, K, r.arg);
      else return launch_vec(k_aa_f32v<false, false, false>, k_aa_f32v<false, false, true>, a.g, r, a.g.nz, st, pf, a.g, K, r.arg);
    }
  }
  // FP16 (automatic or 4): four cells per thread. The automatic BGK odd step has
  // eight where rows are whole chunks: on B200 the pair of AA steps measured
  // 84.3 GLUPS at 256^3 and 86.0 at 512^3 against 80.0 and 81.6 with four cells
  // per thread on both steps; eight cells on the even step as well measured the
  // same (84.1, 86.1), so the even step stays on k_aa_f16v, and eight cells gave
  // the Smagorinsky odd step nothing (76.0 against 76.2, issue-bound). Rows of no
  // power of two: 384 x 256 x 256 85.1 against 56.4 on one cell per thread
  if (F::id == FORM_F16 && (variant == 4 || (variant == 0 && big))) {
    const Pops<__half> ph = pops_of<__half>(a);
    const VecRows r8(a.g, 8, false, true), r(a.g, 4, false);
    if (K.les) {
      if (odd) return launch_vec(k_aa_f16v<true, true, false>, k_aa_f16v<true, true, true>, a.g, r, a.g.nz, st, ph, a.g, K, r.arg);
      else return launch_vec(k_aa_f16v<false, true, false>, k_aa_f16v<false, true, true>, a.g, r, a.g.nz, st, ph, a.g, K, r.arg);
    } else if (odd && variant == 0 && r8.arg >= 0) {
      return launch_vec(k_aa_f16w<true, false>, k_aa_f16w<true, true>, a.g, r8, a.g.nz, st, ph, a.g, K, r8.arg);
    } else {
      if (odd) return launch_vec(k_aa_f16v<true, false, false>, k_aa_f16v<true, false, true>, a.g, r, a.g.nz, st, ph, a.g, K, r.arg);
      else return launch_vec(k_aa_f16v<false, false, false>, k_aa_f16v<false, false, true>, a.g, r, a.g.nz, st, ph, a.g, K, r.arg);
    }
  }
  if (K.les) {
    if (odd) return launch_step(k_aa<F, true, true>, sh.grid, sh.block, st, pops_of<S>(a), a.g, K);
    else return launch_step(k_aa<F, false, true>, sh.grid, sh.block, st, pops_of<S>(a), a.g, K);
  }
  if (variant == 8) {
    bool launched = false;
    cudaError_t e = launch_rows(a, a, odd ? ROW_AA_ODD : ROW_AA_EVEN, K, st, &launched);
    if (e != cudaSuccess || launched) return e;
  }
  if (odd && F::id == FORM_F16)
    return launch_step(k_aa_f16_odd, sh.grid, sh.block, st, pops_of<__half>(a), a.g, K);
  else if (odd) return launch_step(k_aa<F, true>, sh.grid, sh.block, st, pops_of<S>(a), a.g, K);
  else return launch_step(k_aa<F, false>, sh.grid, sh.block, st, pops_of<S>(a), a.g, K);
}

cudaError_t launch_aa(const Lattice& a, int odd, double omega, double scale, double les_cs, int variant,
                      cudaStream_t st) {
  const StepK K = make_stepk(a.form, omega, scale, les_cs);
  switch (a.form) {
    case FORM_F64: return aa_impl<F64>(a, odd, K, variant, st);
    case FORM_F32: return aa_impl<F32>(a, odd, K, variant, st);
    case FORM_F16: return aa_impl<F16>(a, odd, K, variant, st);
  }
  return cudaErrorInvalidValue;
}

template <class F>
static cudaError_t tgv_impl(const Lattice& a, int lay, double u0, int faithful, double scale, unsigned int* mx,
                            cudaStream_t st) {
  using S = typename F::S; using R = typename F::R;
  const long long n = (long long)a.g.nx * a.g.ny * a.g.nz;
  k_init_tgv<F><<<grid_1d(n, 256, 148 * 32), 256, 0, st>>>(pops_of<S>(a), a.g, lay, (R)u0, faithful, (R)scale, mx);
  return cudaGetLastError();
}

cudaError_t launch_init_tgv(const Lattice& a, int lay, double u0, int faithful, double scale, unsigned int* mx,
                            cudaStream_t st) {
  switch (a.form) {
    case FORM_F64: return tgv_impl<F64>(a, lay, u0, faithful, scale, mx, st);
    case FORM_F32: return tgv_impl<F32>(a, lay, u0, faithful, scale, mx, st);
    case FORM_F16: return tgv_impl<F16>(a, lay, u0, faithful, scale, mx, st);
  }
  return cudaErrorInvalidValue;
}

template <class F>
static cudaError_t vel_impl(const Lattice& a, int lay, const double* u, const double* v, const double* w, double rho,
                            int k0, int nk, double scale, unsigned int* mx, cudaStream_t st) {
  using S = typename F::S; using R = typename F::R;
  k_init_vel<F><<<grid_1d(Units(a.g.nx, a.g.ny, nk).n, 8, 148 * 32), 256, 0, st>>>(pops_of<S>(a), a.g, lay, u, v, w, rho, k0, nk, (R)scale,
                                                           mx);
  return cudaGetLastError();
}

cudaError_t launch_init_velocity(const Lattice& a, int lay, const double* u, const double* v, const double* w,
                                 double rho, int k0, int nk, double scale, unsigned int* mx, cudaStream_t st) {
  switch (a.form) {
    case FORM_F64: return vel_impl<F64>(a, lay, u, v, w, rho, k0, nk, scale, mx, st);
    case FORM_F32: return vel_impl<F32>(a, lay, u, v, w, rho, k0, nk, scale, mx, st);
    case FORM_F16: return vel_impl<F16>(a, lay, u, v, w, rho, k0, nk, scale, mx, st);
  }
  return cudaErrorInvalidValue;
}

static int unit_grid(const Geo& g) { return grid_1d(Units(g.nx, g.ny, g.nz).n, 8, 148 * 32); }

template <class F, int LAY>
static void export_lay(const Lattice& a, int q0, int nq, void* ds, double* dd, double scale, cudaStream_t st) {
  using S = typename F::S; using R = typename F::R;
  k_export<F, LAY><<<unit_grid(a.g), 256, 0, st>>>(pops_of<const S>(a), a.g, q0, nq, (S*)ds, dd, (R)(1.0 / scale));
}
template <class F>
static cudaError_t export_impl(const Lattice& a, int lay, int q0, int nq, void* ds, double* dd, double scale,
                               cudaStream_t st) {
  if (lay == LAY_TWO) export_lay<F, LAY_TWO>(a, q0, nq, ds, dd, scale, st);
  else if (lay == LAY_AAE) export_lay<F, LAY_AAE>(a, q0, nq, ds, dd, scale, st);
  else export_lay<F, LAY_AAN>(a, q0, nq, ds, dd, scale, st);
  return cudaGetLastError();
}
cudaError_t launch_export(const Lattice& a, int lay, int q0, int nq, void* ds, double* dd, double scale,
                          cudaStream_t st) {
  switch (a.form) {
    case FORM_F64: return export_impl<F64>(a, lay, q0, nq, ds, dd, scale, st);
    case FORM_F32: return export_impl<F32>(a, lay, q0, nq, ds, dd, scale, st);
    case FORM_F16: return export_impl<F16>(a, lay, q0, nq, ds, dd, scale, st);
  }
  return cudaErrorInvalidValue;
}

template <class F, int LAY>
static void import_lay(const Lattice& a, int q0, int nq, const void* ds, cudaStream_t st) {
  using S = typename F::S;
  k_import<F, LAY><<<unit_grid(a.g), 256, 0, st>>>(pops_of<S>(a), a.g, q0, nq, (const S*)ds);
}
template <class F>
static cudaError_t import_impl(const Lattice& a, int lay, int q0, int nq, const void* ds, cudaStream_t st) {
  if (lay == LAY_TWO) import_lay<F, LAY_TWO>(a, q0, nq, ds, st);
  else if (lay == LAY_AAE) import_lay<F, LAY_AAE>(a, q0, nq, ds, st);
  else import_lay<F, LAY_AAN>(a, q0, nq, ds, st);
  return cudaGetLastError();
}
cudaError_t launch_import(const Lattice& a, int lay, int q0, int nq, const void* ds, cudaStream_t st) {
  switch (a.form) {
    case FORM_F64: return import_impl<F64>(a, lay, q0, nq, ds, st);
    case FORM_F32: return import_impl<F32>(a, lay, q0, nq, ds, st);
    case FORM_F16: return import_impl<F16>(a, lay, q0, nq, ds, st);
  }
  return cudaErrorInvalidValue;
}

template <class S> static Halo<S> halo_of(const SlabLinks* l) {
  Halo<S> h{};
  if (!l) return h;
  for (int s = 0; s < NZF; ++s) {
    h.in_lo[s] = (const S*)l->in_lo[s];
    h.in_hi[s] = (const S*)l->in_hi[s];
    h.up[s] = (S*)l->up[s];
    h.dn[s] = (S*)l->dn[s];
  }
  return h;
}

template <class F, int LAY, int PULL>
static cudaError_t diag_pull(bool overlap, const Lattice& a, double svisc, double omega, double scale, double* partials, void* vel,
                      const SlabLinks* halo, const void* faith, bool fzero, cudaStream_t st) {
  using S = typename F::S; using R = typename F::R;
  return launch_after(overlap, k_diag<F, LAY, PULL>, diag_blocks(F::id), DIAG_THREADS, st, pops_of<const S>(a), a.g,
                      svisc, omega, (R)(1.0 / scale), partials, (R*)vel, halo_of<S>(halo), (const S*)faith,
                      fzero ? 1 : 0);
}
template <class F>
static cudaError_t diag_impl(bool overlap, const Lattice& a, int lay, double svisc, double omega, double scale, double* partials,
                             void* vel, const SlabLinks* halo, const void* faith, bool fzero, cudaStream_t st) {
  if (lay == LAY_AAE) return diag_pull<F, LAY_AAE, PULL_WRAP>(overlap, a, svisc, omega, scale, partials, vel, nullptr, nullptr, false, st);
  if (lay == LAY_AAN) return diag_pull<F, LAY_AAN, PULL_WRAP>(overlap, a, svisc, omega, scale, partials, vel, nullptr, nullptr, false, st);
  if (halo) return diag_pull<F, LAY_TWO, PULL_SLAB>(overlap, a, svisc, omega, scale, partials, vel, halo, nullptr, false, st);
  if (faith || fzero) return diag_pull<F, LAY_TWO, PULL_FAITH>(overlap, a, svisc, omega, scale, partials, vel, nullptr, faith, fzero, st);
  return diag_pull<F, LAY_TWO, PULL_WRAP>(overlap, a, svisc, omega, scale, partials, vel, nullptr, nullptr, false, st);
}

template <class F, class OUT>
static cudaError_t velocity_impl(const Lattice& a, int lay, double scale, void* vel, int k0, int nk,
                                 cudaStream_t st) {
  using S = typename F::S; using R = typename F::R;
  const Units un(a.g.nx, a.g.ny, nk);
  const int grid = grid_1d(un.n, 8, 148 * 32);
  const R inv = (R)(1.0 / scale);
  if (lay == LAY_TWO) k_velocity<F, LAY_TWO, OUT><<<grid, 256, 0, st>>>(pops_of<const S>(a), a.g, inv, (OUT*)vel, k0, nk);
  else if (lay == LAY_AAE) k_velocity<F, LAY_AAE, OUT><<<grid, 256, 0, st>>>(pops_of<const S>(a), a.g, inv, (OUT*)vel, k0, nk);
  else k_velocity<F, LAY_AAN, OUT><<<grid, 256, 0, st>>>(pops_of<const S>(a), a.g, inv, (OUT*)vel, k0, nk);
  return cudaGetLastError();
}
cudaError_t launch_velocity(const Lattice& a, int lay, double scale, void* vel, bool as_double, int k0, int nk,
                            cudaStream_t st) {
  switch (a.form) {
    case FORM_F64: return velocity_impl<F64, double>(a, lay, scale, vel, k0, nk, st);
    case FORM_F32:
      return as_double ? velocity_impl<F32, double>(a, lay, scale, vel, k0, nk, st)
                       : velocity_impl<F32, float>(a, lay, scale, vel, k0, nk, st);
    case FORM_F16:
      return as_double ? velocity_impl<F16, double>(a, lay, scale, vel, k0, nk, st)
                       : velocity_impl<F16, float>(a, lay, scale, vel, k0, nk, st);
  }
  return cudaErrorInvalidValue;
}

long long faith_planes_elems(const Geo& g) {
  return (long long)Q * 2 * ((long long)g.ny * g.nz + (long long)g.nx * g.nz + (long long)g.nx * g.ny);
}

cudaError_t launch_faith_snapshot(const Lattice& a, void* out, cudaStream_t st) {
  const long long n = faith_planes_elems(a.g);
  const int blocks = grid_1d(n, 256, 148 * 16);
  switch (a.form) {
    case FORM_F64: k_faith_snapshot<double><<<blocks, 256, 0, st>>>(pops_of<const double>(a), a.g, (double*)out); break;
    case FORM_F32: k_faith_snapshot<float><<<blocks, 256, 0, st>>>(pops_of<const float>(a), a.g, (float*)out); break;
    case FORM_F16: k_faith_snapshot<__half><<<blocks, 256, 0, st>>>(pops_of<const __half>(a), a.g, (__half*)out); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}
cudaError_t launch_diag(const Lattice& a, int lay, double svisc, double omega, double scale, double* partials,
                        void* vel, cudaStream_t st, const SlabLinks* halo, const void* faith, bool faith_zero,
                        bool overlap) {
  switch (a.form) {
    case FORM_F64: return diag_impl<F64>(overlap, a, lay, svisc, omega, scale, partials, vel, halo, faith, faith_zero, st);
    case FORM_F32: return diag_impl<F32>(overlap, a, lay, svisc, omega, scale, partials, vel, halo, faith, faith_zero, st);
    case FORM_F16: return diag_impl<F16>(overlap, a, lay, svisc, omega, scale, partials, vel, halo, faith, faith_zero, st);
  }
  return cudaErrorInvalidValue;
}

template <class F>
static cudaError_t slab_impl(const Lattice& s, const Lattice& d, const StepK& K, const SlabLinks& l,
                             cudaStream_t st, cudaStream_t st_in) {
  using S = typename F::S;
  Pops<const S> ps = pops_of<const S>(s);
  Pops<S> pd = pops_of<S>(d);
  pd.p[Q - 1] = (S*)s.p[Q - 1];  // pop 19 in place (SRC/col_MC.F90:351)
  const Shape sh = cell_shape(s.g);
  const Halo<S> h = halo_of<S>(&l);
  // planes 0 and nz-1 (one plane when nz = 1) on st, the interior on st_in:
  // the two read only the source lattice and write disjoint planes, so they
  // may run side by side
  const dim3 ge(sh.grid.x, sh.grid.y, s.g.nz > 1 ? 2 : 1);
  if (K.les) k_slab<F, true, true><<<ge, sh.block, 0, st>>>(ps, pd, s.g, K, h);
  else k_slab<F, false, true><<<ge, sh.block, 0, st>>>(ps, pd, s.g, K, h);
  if (s.g.nz > 2) {
    // FP16 / FP32: the interior planes on the four- / two-cells-per-thread
    // kernel (planes 1 .. nz-2 pull only inside the slab, so its z wrap never
    // applies)
    const int ni = s.g.nz - 2;
    const VecRows r(s.g, F::id == FORM_F16 ? 4 : 2, true);
    if (F::id == FORM_F32 && r.pays(s.g, ni)) {
      Pops<float> pf = pops_of<float>(d);
      pf.p[Q - 1] = (float*)s.p[Q - 1];
      if (K.les) launch_vec_plain(k_two_f32v<true, false>, k_two_f32v<true, true>, s.g, r, ni, st_in, pops_of<const float>(s), pf, s.g, K, r.arg, 1);
      else launch_vec_plain(k_two_f32v<false, false>, k_two_f32v<false, true>, s.g, r, ni, st_in, pops_of<const float>(s), pf, s.g, K, r.arg, 1);
    } else if (F::id == FORM_F16 && r.pays(s.g, ni)) {
      Pops<__half> ph = pops_of<__half>(d);
      ph.p[Q - 1] = (__half*)s.p[Q - 1];
      if (K.les) launch_vec_plain(k_two_f16v<true, false>, k_two_f16v<true, true>, s.g, r, ni, st_in, pops_of<const __half>(s), ph, s.g, K, r.arg, 1);
      else launch_vec_plain(k_two_f16v<false, false>, k_two_f16v<false, true>, s.g, r, ni, st_in, pops_of<const __half>(s), ph, s.g, K, r.arg, 1);
    } else {
      const dim3 gi(sh.grid.x, sh.grid.y, s.g.nz - 2);
      if (K.les) k_slab<F, true, false><<<gi, sh.block, 0, st_in>>>(ps, pd, s.g, K, h);
      else k_slab<F, false, false><<<gi, sh.block, 0, st_in>>>(ps, pd, s.g, K, h);
    }
  }
  return cudaGetLastError();
}

cudaError_t launch_slab(const Lattice& src, const Lattice& dst, const SlabLinks& links, double omega, double scale,
                        double les_cs, cudaStream_t st, cudaStream_t st_interior) {
  const StepK K = make_stepk(src.form, omega, scale, les_cs);
  switch (src.form) {
    case FORM_F64: return slab_impl<F64>(src, dst, K, links, st, st_interior);
    case FORM_F32: return slab_impl<F32>(src, dst, K, links, st, st_interior);
    case FORM_F16: return slab_impl<F16>(src, dst, K, links, st, st_interior);
  }
  return cudaErrorInvalidValue;
}

template <class S>
static cudaError_t prime_impl(const Lattice& a, const SlabLinks& l, cudaStream_t st) {
  const int tx = a.g.nx >= 256 ? 256 : ((a.g.nx + 31) / 32) * 32;
  k_halo_prime<S><<<dim3((a.g.nx + tx - 1) / tx, a.g.ny), tx, 0, st>>>(pops_of<const S>(a), a.g, halo_of<S>(&l));
  return cudaGetLastError();
}

cudaError_t launch_halo_prime(const Lattice& a, const SlabLinks& links, cudaStream_t st) {
  switch (a.form) {
    case FORM_F64: return prime_impl<double>(a, links, st);
    case FORM_F32: return prime_impl<float>(a, links, st);
    case FORM_F16: return prime_impl<__half>(a, links, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_enstrophy(const Lattice& a, const void* vel, double* partials, cudaStream_t st) {
  if (a.form == FORM_F64)
    return launch_step(k_enstrophy<double>, DIAG_BLOCKS, DIAG_THREADS, st, (const double*)vel, a.g.nx, a.g.ny, a.g.nz, partials);
  return launch_step(k_enstrophy<float>, DIAG_BLOCKS, DIAG_THREADS, st, (const float*)vel, a.g.nx, a.g.ny, a.g.nz, partials);
}

cudaError_t launch_finalize(const double* partials, int form, bool enstrophy, double* totals, cudaStream_t st,
                            const int* err, bool overlap) {
  return launch_after(overlap, k_finalize, enstrophy ? ND : NDK, DIAG_THREADS, st, partials, diag_blocks(form), totals, err);
}

template <class F>
static cudaError_t lastzj_impl(const Lattice& a, int lay, double scale, double* out, cudaStream_t st) {
  using S = typename F::S; using R = typename F::R;
  const R inv = (R)(1.0 / scale);
  if (lay == LAY_TWO) k_last_zj<F, LAY_TWO><<<1, 32, 0, st>>>(pops_of<const S>(a), a.g, inv, out);
  else if (lay == LAY_AAE) k_last_zj<F, LAY_AAE><<<1, 32, 0, st>>>(pops_of<const S>(a), a.g, inv, out);
  else k_last_zj<F, LAY_AAN><<<1, 32, 0, st>>>(pops_of<const S>(a), a.g, inv, out);
  return cudaGetLastError();
}
cudaError_t launch_last_zj(const Lattice& a, int lay, double scale, double* out, cudaStream_t st) {
  switch (a.form) {
    case FORM_F64: return lastzj_impl<F64>(a, lay, scale, out, st);
    case FORM_F32: return lastzj_impl<F32>(a, lay, scale, out, st);
    case FORM_F16: return lastzj_impl<F16>(a, lay, scale, out, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_shift3(const void* const in[3], void* const out[3], int nx, int ny, int nz, int elem_bytes,
                          int reverse, cudaStream_t st) {
  const long long n = (long long)nx * ny * nz;
  const int grid = grid_1d(n, 256, 148 * 16);
  const int dir = reverse ? -1 : 1;
  if (elem_bytes == 8)
    k_shift3<double><<<grid, 256, 0, st>>>((const double*)in[0], (const double*)in[1], (const double*)in[2],
                                           (double*)out[0], (double*)out[1], (double*)out[2], nx, ny, nz, dir);
  else if (elem_bytes == 4)
    k_shift3<float><<<grid, 256, 0, st>>>((const float*)in[0], (const float*)in[1], (const float*)in[2],
                                          (float*)out[0], (float*)out[1], (float*)out[2], nx, ny, nz, dir);
  else if (elem_bytes == 2)
    k_shift3<__half><<<grid, 256, 0, st>>>((const __half*)in[0], (const __half*)in[1], (const __half*)in[2],
                                           (__half*)out[0], (__half*)out[1], (__half*)out[2], nx, ny, nz, dir);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

template <class F, int LAY>
static void vtk_lay(const Lattice& a, int kind, int index, float* out, long long npts, double scale,
                    cudaStream_t st) {
  using S = typename F::S; using R = typename F::R;
  k_vtk<F, LAY><<<grid_1d(npts, 256, 148 * 16), 256, 0, st>>>(pops_of<const S>(a), a.g, kind, index, out, npts,
                                                               (R)(1.0 / scale));
}
template <class F>
static cudaError_t vtk_impl(const Lattice& a, int lay, int kind, int index, float* out, long long npts, double scale,
                            cudaStream_t st) {
  if (lay == LAY_TWO) vtk_lay<F, LAY_TWO>(a, kind, index, out, npts, scale, st);
  else if (lay == LAY_AAE) vtk_lay<F, LAY_AAE>(a, kind, index, out, npts, scale, st);
  else vtk_lay<F, LAY_AAN>(a, kind, index, out, npts, scale, st);
  return cudaGetLastError();
}
cudaError_t launch_vtk(const Lattice& a, int lay, int kind, int index, float* out, long long npts, double scale,
                       cudaStream_t st) {
  switch (a.form) {
    case FORM_F64: return vtk_impl<F64>(a, lay, kind, index, out, npts, scale, st);
    case FORM_F32: return vtk_impl<F32>(a, lay, kind, index, out, npts, scale, st);
    case FORM_F16: return vtk_impl<F16>(a, lay, kind, index, out, npts, scale, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace bgk
