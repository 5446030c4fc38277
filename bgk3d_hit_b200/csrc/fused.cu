// Two consecutive two-lattice steps in one pass over the populations (k_two2).
//
// A single step moves every population twice (304 bytes a cell in FP64) and is
// bound by that. k_two2 reads a state once and writes the state two steps later:
// a block owns a tile of 32 x TY cells of a plane and walks up z. Its first warps
// take the 34 x (TY + 2) cells of the tile and its border through the first step,
// one plane per interval, into shared memory; the others pull from there and take
// the 32 x TY cells of the tile through the second step. Per plane a thread of
// the second step needs the cz = +1 populations of the plane below, the cz = 0
// ones of its own plane and the cz = -1 ones of the plane above, so it keeps the
// first fourteen in registers until the third plane is there, and shared memory
// holds the post-collision populations of two planes only (one being written,
// one being read). The border is computed by both tiles that share it: a third
// more first-step collisions in x and y (TY = 8), two planes per walk in z. Each
// cell's arithmetic is F::cell's, so two fused steps give the bits of two single
// ones.
//
// The raw planes come by TMA, one box of 36 x (TY + 2) values per population, two
// planes ahead of their use, issued by a warp of its own. Tiles at an x face get
// the periodic columns by a second, 32-byte wide box beside the first; rows beyond
// a y face, which TMA fills with zeros, are put in by the threads.
//
// Measured on B200 at 256^3 FP64 (two steps): 944 us, 35.5 GLUPS, over 20 steps at full
// clock; 1058-1107 us in runs of some tenths of a second, once the power limit lowers
// the clock; against 1515-1524 us (22.1, the HBM rate) for two single steps. DRAM 305 bytes
// a cell for both, FP64 pipe 51% busy, issue slots 47%. What stands between it and the
// 43 GLUPS of its DRAM bytes is the interval (1.1 us of FP64 pipe, one barrier of all
// warps per plane). Figures of single variants below and at the rules are from the
// kernel as it stood then, both sides alike. On the way there: both steps by the same warps 25.6 GLUPS (too few warps between barriers), one raw buffer
// 25.5 (the load of a plane did not fit beside its predecessor's collisions), loads
// of 8 bytes by cp.async 25.6, the border of all faces patched by the threads
// 31.2, the boxes issued by a warp that also collides 28.7-31.2, arrive / wait
// barriers instead of the common one 29.3.
#include <cuda.h>

#include "kernels.h"
#include "launch.cuh"

namespace bgk {

namespace {

constexpr int TX = 32;         // cells of a tile's row: one warp
constexpr int PITCH = TX + 2;  // and of its first step, with the border
constexpr int MAX_POLLS = 1 << 16;  // of POLL_NS each at most: about a second
constexpr int POLL_NS = 1 << 14;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bounded: false when the copies did not land.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int polls) {
  for (int n = 0; n < polls; ++n) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done)
                 : "r"(bar), "r"(parity), "r"(POLL_NS)
                 : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void tma_box(uint32_t dst, const CUtensorMap* m, int x, int y, int z, int q, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
          dst),
      "l"(m), "r"(x), "r"(y), "r"(z), "r"(q), "r"(bar)
      : "memory");
}

__device__ __forceinline__ int modw(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}

template <class S, int TY> struct Two2 {
  static constexpr int ROWS = TY + 2;
  static constexpr int HALO = (2 * ROWS + 31) / 32;           // warps of border columns
  static constexpr int ATH = 32 * (ROWS + HALO);              // threads of the first step
  static constexpr int WORK = ATH + 32 * TY;                  // and of the second
  static constexpr int THREADS = WORK + 32;                   // and a warp that issues the loads
  static constexpr int PAD = 16 / (int)sizeof(S);             // columns before the tile: boxes start on 16 bytes
  static constexpr int RP = (PAD + TX + 2 + PAD - 1) / PAD * PAD;  // row of a main box
  static constexpr int WP = 2 * PAD;                          // row of a wrap box
  static constexpr int W0 = (RP * ROWS * (int)sizeof(S) + 127) / 128 * 128 / (int)sizeof(S);  // wrap box in a block
  static constexpr int RAW = W0 + (WP * ROWS * (int)sizeof(S) + 127) / 128 * 128 / (int)sizeof(S);
  static constexpr int YROWS = 19;                            // raw rows beyond a y face, at most
  static constexpr int YCOLS = TX + 4;                        // columns of a raw row that are read
  static constexpr int NPE = (YROWS * YCOLS + ATH - 1) / ATH; // their elements per thread
  struct Smem {
    S raw[2][Q][RAW];
    S post[2][Q][ROWS * PITCH];
    const S* base[Q];
    int yrow[YROWS], yrq[YROWS];  // plane offset of the row that stands for raw row r of population q; q * 64 + r
    unsigned long long bar[2];
    int failed;  // a wait for a plane ran out
  };
};

// Populations 0..17 of a lattice follow each other; the rest population (18) of the
// time loop's lattices may lie elsewhere and has maps of its own.
struct Two2Maps { CUtensorMap main, wrap, rest_main, rest_wrap; };

// First plane of walk i: `full` walks of lz planes, then half of what is left at a
// time, the last walk taking the rest.
__device__ __forceinline__ int walk_begin(int i, int nz, int lz, int full) {
  const int rest = nz - full * lz;
  return i <= full ? i * lz : full * lz + rest - (rest >> (i - full));
}

template <class F, bool LES, int TY>
__global__ void __launch_bounds__(Two2<typename F::S, TY>::THREADS, 1)
    k_two2(const __grid_constant__ Two2Maps maps, Pops<const typename F::S> src, Pops<typename F::S> dst, Geo g,
           StepK K, int lz, int full, int* err, int stall) {
  using S = typename F::S;
  using T = Two2<S, TY>;
  constexpr int ROWS = T::ROWS;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  typename T::Smem& sm = *reinterpret_cast<typename T::Smem*>(smem_raw);
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  // the last tiles in y move down to end with the box: rows shared with their
  // neighbours are written twice, with the same bits
  const int x0 = blockIdx.x * TX, y0 = min((int)blockIdx.y * TY, g.ny - TY);
  const int z0 = walk_begin(blockIdx.z, g.nz, lz, full);
  const int lzc = ((int)blockIdx.z + 1 < (int)gridDim.z ? walk_begin(blockIdx.z + 1, g.nz, lz, full) : g.nz) - z0;
  const int txc = min(TX, g.nx - x0);
  const int plane = g.sx * g.ny;
  const int np = lzc + 2;                                    // first-step planes
  const bool left = x0 == 0, right = x0 + TX + 2 > g.nx;     // never both (nx >= 34)
  const int beyond = g.ny - (y0 + TY);                       // rows between the tile and the upper y face
  const bool yedge = y0 == 0 || beyond < 2;

  auto issue = [&](int k, int z) {  // plane z into buffer k & 1
    const uint32_t bar = smem_u32(&sm.bar[k & 1]);
    const int zm = z == 0 ? g.nz - 1 : z - 1, zp = z == g.nz - 1 ? 0 : z + 1;
    const int xw = left ? (g.nx - 2) / T::PAD * T::PAD : 0;
    // the buffer was read and patched by ordinary accesses before this
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                 "r"((uint32_t)(Q * ROWS * (T::RP + (left || right ? T::WP : 0)) * (int)sizeof(S)))
                 : "memory");
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int zz = czq(q) > 0 ? zm : (czq(q) < 0 ? zp : z), qq = q == Q - 1 ? 0 : q;
      const uint32_t d = smem_u32(&sm.raw[k & 1][q][0]);
      tma_box(d, q == Q - 1 ? &maps.rest_main : &maps.main, x0 - T::PAD, y0 - 1 - cyq(q), zz, qq, bar);
      if (left || right)
        tma_box(d + T::W0 * (int)sizeof(S), q == Q - 1 ? &maps.rest_wrap : &maps.wrap, xw, y0 - 1 - cyq(q), zz, qq, bar);
    }
  };
  auto next = [&](int p) { return p == g.nz - 1 ? 0 : p + 1; };

  // test hook: the first block's first plane is never asked for
  const bool stalled = stall && (blockIdx.x | blockIdx.y | blockIdx.z) == 0;

  // nothing of the step before is read or overwritten before it is done
  step_begin();

  if (tid == T::WORK) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sm.bar[0])) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&sm.bar[1])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    const int z = modw(z0 - 1, g.nz);
    sm.failed = 0;
    if (!stalled) issue(0, z);
    issue(1, next(z));
  }
  int yn = 0;  // raw rows beyond the y face
  if (yedge) {
    int n = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (tid == q) sm.base[q] = src.p[q];
      // lower face: rows -2 and -1 of cy = 1, row -1 of cy = 0; upper: mirrored
      const int rows = y0 == 0 ? 1 + cyq(q) : max(0, 1 - cyq(q) - beyond);
      if (tid >= n && tid < n + rows) {
        const int r = y0 == 0 ? tid - n : ROWS - 1 - (tid - n);
        sm.yrow[tid] = g.sx * modw(y0 + r - 1 - cyq(q), g.ny);
        sm.yrq[tid] = q * 64 + r;
      }
      n += rows;
    }
    yn = n;
  }
  __syncthreads();

  // interval k: the first step of plane k beside the second step around plane k - 1
  if (w == T::WORK / 32) {
    int z = next(next(modw(z0 - 1, g.nz)));
    // (The form of this loop matters: with its bound at np - 2, or ok preset where the
    // test hook leaves out plane 0, the same launches are 2-5% slower, us per pair FP64
    // 256^3 1057 / 1086-1104, FP32 180^3 246 / 246-257.)
    int asked = 1;  // last plane asked for
    bool ok = true;
    for (int k = 0; k < np; ++k, z = next(z)) {
      if (stalled && k == 0) ok = false;
      if (k + 2 >= np) continue;
      // Plane k has been read. Two barriers in turn: a warp comes to plane k + 2,
      // which this warp asks for below, only after this wait is over, but may come
      // to plane k + 1 before this warp comes here, and must not count for plane k
      asm volatile("bar.sync %0, %1;" ::"r"(4 + (k & 1)), "n"(T::ATH + 32) : "memory");
      // Or it has not come: its copies may still be under way, and its buffer's barrier
      // is in their phase
      if (*(volatile int*)&sm.failed) ok = false;
      if (ok) {
        if (lane == 0) issue(k, z);
        asked = k + 2;
      }
      __syncwarp();
    }
    // No copy may reach the shared memory of a block that has ended. The first step's
    // warps have waited for all planes unless one of their waits ran out.
    for (int k = stalled ? 1 : asked - 1; k <= asked; ++k)
      (void)mbar_wait(smem_u32(&sm.bar[k & 1]), (k >> 1) & 1, MAX_POLLS);
  } else if (tid < T::ATH) {
    int r, c;  // first-step cell of this thread: row, column of the tile (-1 .. 32)
    if (w < ROWS) {
      r = w;
      c = lane;
    } else {
      const int h = (w - ROWS) * 32 + lane;
      r = h >> 1;
      c = (h & 1) ? TX : -1;
    }
    const bool on = r < ROWS;
    const int slot = r * PITCH + c + 1;
    // element of a block that holds column c + d of the row, d = -1, 0, 1
    auto elem = [&](int row, int col) {
      if (left && col < 0) return T::W0 + row * T::WP + col + g.nx - (g.nx - 2) / T::PAD * T::PAD;
      if (right && x0 + col >= g.nx) return T::W0 + row * T::WP + min(x0 + col - g.nx, T::WP - 1);
      return row * T::RP + T::PAD + col;
    };
    const int em = elem(r, c - 1), e0 = elem(r, c), ep = elem(r, c + 1);
    // rows beyond a y face: this thread's elements of the plane to come
    S yv[T::NPE];
    int zy = modw(z0 - 1, g.nz);
    auto load_y = [&]() {
      const int zc = zy * plane, zm = (zy == 0 ? g.nz - 1 : zy - 1) * plane, zp = (zy == g.nz - 1 ? 0 : zy + 1) * plane;
#pragma unroll
      for (int m = 0; m < T::NPE; ++m) {
        const int e = tid + m * T::ATH, n = e / T::YCOLS;
        if (n < yn) {
          const int q = sm.yrq[n] >> 6, cz = czq(q);
          yv[m] = sm.base[q][sm.yrow[n] + modw(x0 + e % T::YCOLS - 2, g.nx) + (cz > 0 ? zm : (cz < 0 ? zp : zc))];
        }
      }
      zy = next(zy);
    };
    if (yedge) load_y();
    bool dead = false;
    for (int k = 0; k < np; ++k) {
      S* const raw = &sm.raw[k & 1][0][0];
      // After a wait that ran out the state is invalid, which is reported; the warp goes
      // through its remaining intervals on whatever the planes hold.
      if (!mbar_wait(smem_u32(&sm.bar[k & 1]), (k >> 1) & 1, dead ? 1 : MAX_POLLS)) {
        dead = true;
        *(volatile int*)&sm.failed = 1;
        *err = 1;
        __threadfence_block();
      }
      __syncwarp();
      if (yedge) {
#pragma unroll
        for (int m = 0; m < T::NPE; ++m) {
          const int e = tid + m * T::ATH, n = e / T::YCOLS;
          if (n < yn) raw[(sm.yrq[n] >> 6) * T::RAW + elem(sm.yrq[n] & 63, e % T::YCOLS - 2)] = yv[m];
        }
        asm volatile("bar.sync 2, %0;" ::"n"(T::ATH) : "memory");
        if (k + 1 < np) load_y();
      }
      S v[Q];
      if (on) {
#pragma unroll
        for (int q = 0; q < Q; ++q) v[q] = raw[q * T::RAW + (cxq(q) > 0 ? em : (cxq(q) < 0 ? ep : e0))];
      }
      __syncwarp();
      if (k + 2 < np) asm volatile("bar.arrive %0, %1;" ::"r"(4 + (k & 1)), "n"(T::ATH + 32) : "memory");
      if (on) {
        F::template cell<LES>(v, K);
        S* const b = sm.post[k & 1][0];
#pragma unroll
        for (int q = 0; q < Q; ++q) b[q * ROWS * PITCH + slot] = v[q];
      }
      asm volatile("bar.sync 3, %0;" ::"n"(T::WORK) : "memory");
    }
  } else {
    const int r = w - T::ATH / 32 + 1;  // row of output cells, 1 .. TY
    const bool st = lane < txc;
    const int slot = r * PITCH + lane + 1;
    S P1[NZF], N1[NZF], C0[Q - 2 * NZF];  // cz = +1 of the last plane but one and the last, cz = 0 of the last
#pragma unroll
    for (int m = 0; m < NZF; ++m) P1[m] = N1[m] = S(0.f);
#pragma unroll
    for (int m = 0; m < Q - 2 * NZF; ++m) C0[m] = S(0.f);
    int o = x0 + lane + g.sx * (y0 + r - 1) + z0 * plane;  // next output cell
    for (int k = 0; k < np; ++k) {
      asm volatile("bar.sync 3, %0;" ::"n"(T::WORK) : "memory");
      const S* const b = sm.post[k & 1][0];
      auto pull = [&](int q) { return b[q * ROWS * PITCH + slot - cyq(q) * PITCH - cxq(q)]; };
      if (k >= 2) {
        S v[Q];
        int n = 0;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          if (czq(q) > 0) v[q] = P1[zslot(q)];
          else if (czq(q) == 0) v[q] = C0[n++];
          else v[q] = pull(q);
        }
        F::template cell<LES>(v, K);
        if (st) {
#pragma unroll
          for (int q = 0; q < Q; ++q) dst.p[q][o] = v[q];
        }
        o += plane;
      }
      int n = 0;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (czq(q) > 0) {
          P1[zslot(q)] = N1[zslot(q)];
          N1[zslot(q)] = pull(q);
        } else if (czq(q) == 0) {
          C0[n++] = pull(q);
        }
      }
    }
  }
}

template <class S> Pops<S> pops(const Lattice& L) {
  Pops<S> p;
  for (int q = 0; q < Q; ++q) p.p[q] = (S*)L.p[q];
  return p;
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                             const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Tensor map of nq populations that follow each other every qs elements.
bool encode(CUtensorMap* m, const Geo& g, int form, void* base, int nq, int cols, int rows) {
  static const EncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &r) != cudaSuccess) p = nullptr;
    return (EncodeFn)p;
  }();
  if (!fn) return false;
  const int es = form == FORM_F64 ? 8 : (form == FORM_F32 ? 4 : 2);
  const cuuint64_t dims[4] = {(cuuint64_t)g.nx, (cuuint64_t)g.ny, (cuuint64_t)g.nz, (cuuint64_t)nq};
  const cuuint64_t str[3] = {(cuuint64_t)g.sx * es, (cuuint64_t)g.sx * g.ny * es, (cuuint64_t)g.qs * es};
  const cuuint32_t box[4] = {(cuuint32_t)cols, (cuuint32_t)rows, 1, 1}, one[4] = {1, 1, 1, 1};
  const CUtensorMapDataType dt = form == FORM_F64 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64
                                 : form == FORM_F32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  return fn(m, dt, 4, base, dims, str, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Height of the tiles: what registers and shared memory of an SM hold. FP64: 20
// warps at 96 registers, no spills (BGK); the Smagorinsky collision needs 120
// (TY = 6, 16 warps; at TY = 8 244 bytes spill and 256^3 takes 1408 us instead of
// 1271). FP32: the 1024 threads of a block (TY = 12: 706 us instead of 649).
template <class F, bool LES> constexpr int tile_rows() { return F::id == FORM_F64 ? (LES ? 6 : 8) : 14; }

constexpr int SMS = 148;

// How a column of tiles is cut into walks. Planes per walk: the sum of all walks (each
// two planes longer than what it writes) over the SMs, and one walk for the uneven
// end, in intervals, are least (256^3 FP64, 256 tiles: 32 planes 998 us, 16 1023, 64
// 1044). The last walk is halved twice, so that the SMs that are done first are not idle
// for a whole walk: equal walks / halved, us per two steps of long runs, FP32 256^3 693 /
// 677, 180^3 271 / 265, 160^3 192 / 189; FP64 256^3 1136 / 1127, 128^3 174.9 / 173.6;
// Smagorinsky 256^3 1419 / 1418.
struct Walks {
  int lz, full, halvings;
  double tiles;
  int nz;
  Walks(const Geo& g, int ty)
      : lz(g.nz), tiles((double)((g.nx + TX - 1) / TX) * ((g.ny + ty - 1) / ty)), nz(g.nz) {
    double least = 1e300;
    for (int n = 1; n <= nz; ++n) {
      const int l = (nz + n - 1) / n, walks = (nz + l - 1) / l;
      const double c = tiles * walks * (l + 2) / SMS + (l + 2);
      if (c < least) {
        least = c;
        lz = l;
      }
    }
    full = (nz + lz - 1) / lz - 1;
    halvings = nz - full * lz >= 4 ? 2 : 0;
  }
  int count() const { return full + 1 + halvings; }
  // Of the whole launch: what all walks take, spread over the SMs, and half a walk for
  // the end. A walk costs its planes, two more that it does not write, and about half
  // an interval to start; flat boxes, whose walks are a few planes long, pay the most.
  double intervals() const { return tiles * (nz + count() * 2.5) / SMS + 0.5 * (lz + 2.5); }
};

template <class F, bool LES>
cudaError_t launch(const Lattice& s, const Lattice& d, const StepK& K, cudaStream_t st) {
  using S = typename F::S;
  constexpr int TY = tile_rows<F, LES>();
  using T = Two2<S, TY>;
  constexpr size_t bytes = sizeof(typename T::Smem);
  static_assert(bytes <= 232448 && T::THREADS <= 1024, "an SM's shared memory and a block's threads");
  const auto kern = k_two2<F, LES, TY>;
  const Geo& g = s.g;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  Two2Maps m;
  if (!encode(&m.main, g, s.form, s.p[0], Q - 1, T::RP, T::ROWS) ||
      !encode(&m.wrap, g, s.form, s.p[0], Q - 1, T::WP, T::ROWS) ||
      !encode(&m.rest_main, g, s.form, s.p[Q - 1], 1, T::RP, T::ROWS) ||
      !encode(&m.rest_wrap, g, s.form, s.p[Q - 1], 1, T::WP, T::ROWS))
    return cudaErrorInvalidValue;
  const Walks w(g, TY);
  const dim3 grid((g.nx + TX - 1) / TX, (g.ny + TY - 1) / TY, w.count());
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(T::THREADS);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, m, pops<const S>(s), pops<S>(d), g, K, w.lz, w.full, s.err, s.stall);
}

}  // namespace

// An interval of the launch takes about 2.0 us (1.85-2.2 over the boxes below), a
// single step the time of its cells at the rate given. Runs of 0.7 s, us per two steps,
// two per launch / single steps:
//   FP64 80^3 63 / 51, 96^3 78 / 86, 112^3 124 / 139, 128^3 166 / 194, 256^3 1058 / 1524,
//     250 x 130 x 130 321 / 393, 512 x 512 x 8 224 / 193 and x 16 349 / 385, 1024 x 1024 x
//     4 645 / 388;
//   Smagorinsky 112^3 154 / 153, 128^3 198 / 207, 160^3 364 / 468, 256^3 1369 / 1619, 64 x 64 x
//     512 209 / 207, 512 x 512 x 8 320 / 206 and x 32 788 / 836;
//   FP32 128^3 107 / 102, 140^3 135 / 148, 160^3 180 / 197, 180^3 251 / 300, 256^3 632 / 770,
//     1024 x 1024 x 8 499 / 396.
// Of 97 boxes measured so, the rule takes two that lose 1%, and leaves nine at single
// steps that would gain 2-8% (one 16%). Not built: FP32 Smagorinsky (734 / 757 at 256^3,
// 306 / 298 at 180^3, short runs) and FP16, whose single step runs at the copy rate
// already (86 GLUPS, against 51 and 64 here).
bool two_steps_pay(const Geo& g, int form, bool les) {
  if (form != FORM_F64 && (form != FORM_F32 || les)) return false;
  const int ty = form == FORM_F64 ? (les ? 6 : 8) : 14;
  // a tile touches one x face and one y face at most; TMA sizes and strides
  if (g.nx < TX + 2 || g.ny < ty + 2) return false;
  const bool aligned = (g.nx & (g.nx - 1)) == 0;
  const double rate = form == FORM_F32 ? (aligned ? 43.5e3 : 38.5e3)
                      : les ? (aligned ? 20e3 : 18.5e3) : (aligned ? 21.5e3 : 20.5e3);  // cells per us
  return 2.0 * Walks(g, ty).intervals() < 2.0 * (double)g.nx * g.ny * g.nz / rate;
}

cudaError_t launch_two_steps(const Lattice& src, const Lattice& dst, double omega, double scale, double les_cs,
                             cudaStream_t st) {
  const StepK K = make_stepk(src.form, omega, scale, les_cs);
  if (src.form == FORM_F64) return K.les ? launch<F64, true>(src, dst, K, st) : launch<F64, false>(src, dst, K, st);
  if (src.form == FORM_F32 && !K.les) return launch<F32, false>(src, dst, K, st);
  return cudaErrorInvalidValue;
}

}  // namespace bgk
