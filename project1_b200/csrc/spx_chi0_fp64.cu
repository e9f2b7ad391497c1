// K1, K1p, K1r: FP64 band-pair accumulation on the DMMA tensor path (the drop-in).
//
// Most calls run on the product-first kernels further down (K1p: complex, -DINV and the
// q -> 0 head and wings); the two that follow the sum frequency by frequency keep calls of
// few frequencies or few pairs where they are faster (f64_on_k1). K1 computes,
// for every upper-triangle 64x64 tile (I, J) of the mixed-basis
// matrix and every frequency f,
//   chi_f(i, j) += sum_p M(p, i) * conj(M(p, j)) * w(p, f),      i <= j,
// which is the body loop of src/susceptibility.f:1182-1240 with the HILBERT
// NONE spectral_function (:1766-1789) folded in: the reference forms
// re/im(k) = cprod(k,i)*conjg(cprod(k,j)) for one (i,j) at a time and takes a
// ddot per frequency; here the same sum is a weighted complex Gram evaluated
// tile by tile, so every loaded band-pair value feeds 64 outputs instead of one.
//
// Layout and pipeline:
//   * one work item = (frequency, upper tile); persistent CTAs stride over items;
//   * warp 0 streams 16-pair slabs of the two 64-column panels of M
//     (p-contiguous columns, exactly the Fortran cprod layout) into shared memory
//     with 2-D TMA boxes of 8 pairs x 64 columns (128-byte rows, SWIZZLE_128B, so
//     fragment loads of eight rows hit eight different bank groups), three stages
//     ahead (five copy instructions per stage); pairs and columns past the slab's
//     end arrive as zeros, and a diagonal tile loads its one panel once;
//   * four warps each own a 32x32 complex sub-tile and run
//     mma.sync m16n8k8 f64 on re/im parts: re += ar*(w br) + ai*(w bi),
//     im += ai*(w br) - ar*(w bi); each warp releases a stage on an mbarrier;
//   * the epilogue adds the tile into the packed upper triangle
//     susceph(j*(j+1)/2 + i, f) (src/susceptibility.f:1210).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "spx_common.cuh"
#include "spx_dmma.cuh"
#include "spx_tcgen05.cuh"

namespace spx {

constexpr int F64_B = 64;                 // tile edge in complex rows / columns
constexpr int F64_KC = 16;                // band pairs per pipeline stage
constexpr int F64_KBOX = 8;               // pairs per TMA box: one 128-byte swizzled row
constexpr int F64_ST = 3;                 // pipeline stages
constexpr int F64_WARPS = 4;              // each owns a 32x32 complex sub-tile
constexpr int F64_THREADS = 32 * F64_WARPS;

struct F64Params {
  int64_t P;
  int N;
  const double* W;
  int64_t ldw;
  int nw;
  double2* out;
  int64_t npack;
  int ntile;
  int64_t nitems;
  int* status;
  uint64_t timeout_ns;
};

// one panel half: 64 columns x 8 pairs, row r's 16-byte chunk c stored at c ^ (r & 7)
typedef double2 F64Box[F64_B][F64_KBOX];

struct __align__(1024) F64Smem {
  F64Box a[F64_ST][2];
  F64Box b[F64_ST][2];
  double w[F64_ST][F64_KC];
  uint64_t full[F64_ST];
  uint64_t empty[F64_ST];  // every compute warp has finished with the stage
};

// Upper-triangle tile t -> (bi, bj), bi <= bj, column-major over the triangle.
__device__ __forceinline__ void decode_tile(int t, int* bi, int* bj) {
  int j = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while (j * (j + 1) / 2 > t) --j;
  while ((j + 1) * (j + 2) / 2 <= t) ++j;
  *bj = j;
  *bi = t - j * (j + 1) / 2;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

__global__ void __launch_bounds__(F64_THREADS, 2)
    chi0_fp64_kernel(const __grid_constant__ CUtensorMap mapM, F64Params prm) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  F64Smem& sm = *reinterpret_cast<F64Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                            ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < F64_ST; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], F64_WARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();

  // The chunk sequence of this CTA: items blockIdx.x, +gridDim.x, ...; each item
  // is nchunk slabs of F64_KC band pairs. Chunk c lives in stage c % F64_ST.
  const int64_t nchunk = (prm.P + F64_KC - 1) / F64_KC;
  const int64_t my_items = prm.nitems > blockIdx.x
                               ? (prm.nitems - blockIdx.x + gridDim.x - 1) / gridDim.x
                               : 0;
  const int64_t total = my_items * nchunk;
  auto chunk_item = [&](int64_t c) { return blockIdx.x + (c / nchunk) * (int64_t)gridDim.x; };
  auto chunk_p0 = [&](int64_t c) { return (c % nchunk) * (int64_t)F64_KC; };

  // chunk c's copies (one thread): 2 or 4 boxes of M and the 16 weights
  auto issue = [&](int64_t c) {
    const int st = (int)(c % F64_ST);
    const int64_t item = chunk_item(c), p0 = chunk_p0(c);
    const int f = (int)(item / prm.ntile);
    int bi, bj;
    decode_tile((int)(item % prm.ntile), &bi, &bj);
    const bool same = bi == bj;
    mbar_arrive_expect_tx(&sm.full[st], (uint32_t)((same ? 2 : 4) * sizeof(F64Box) + F64_KC * 8));
    const int x = (int)(2 * p0);
    tma_load_2d(&sm.a[st][0][0][0], &mapM, x, bi * F64_B, &sm.full[st]);
    tma_load_2d(&sm.a[st][1][0][0], &mapM, x + 2 * F64_KBOX, bi * F64_B, &sm.full[st]);
    if (!same) {
      tma_load_2d(&sm.b[st][0][0][0], &mapM, x, bj * F64_B, &sm.full[st]);
      tma_load_2d(&sm.b[st][1][0][0], &mapM, x + 2 * F64_KBOX, bj * F64_B, &sm.full[st]);
    }
    bulk_g2s(&sm.w[st][0], prm.W + (int64_t)f * prm.ldw + p0, F64_KC * 8, &sm.full[st]);
  };
  // chunks [0, issued) have their copies issued (tracked by warp 0, lane 0)
  int64_t issued = total < F64_ST - 1 ? total : (int64_t)(F64_ST - 1);
  if (warp == 0 && lane == 0)
    for (int64_t c = 0; c < issued; ++c) issue(c);

  // ---------------- compute warps ----------------
  const int wi = warp & 1, wj = warp >> 1;
  const int g = lane >> 2, t = lane & 3;
  double accR[2][4][4], accI[2][4][4];
  bool failed = false;
  int64_t c = 0;
  for (; c < total; ++c) {
    const int st = (int)(c % F64_ST);
    const uint32_t ph = (uint32_t)((c / F64_ST) & 1);
    const int64_t item = chunk_item(c), p0 = chunk_p0(c);
    int bi, bj;
    decode_tile((int)(item % prm.ntile), &bi, &bj);
    if (p0 == 0) {
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int r = 0; r < 4; ++r) accR[mt][nt][r] = accI[mt][nt][r] = 0.0;
    }
    // chunk c + F64_ST - 1 goes into the stage of chunk c - 1, once all four warps
    // have released that one (its release completes phase (c-1)/F64_ST of empty)
    if (warp == 0 && c + F64_ST - 1 < total) {
      const int64_t prev = c - 1;
      int ok = 1;
      if (lane == 0) {
        if (prev >= 0)
          ok = mbar_wait(&sm.empty[(int)(prev % F64_ST)], (uint32_t)((prev / F64_ST) & 1),
                         prm.timeout_ns, prm.status);
        if (ok) issue(c + F64_ST - 1);
      }
      if (!__shfl_sync(0xffffffffu, ok, 0)) {
        failed = true;
        break;
      }
      issued = c + F64_ST;
    }
    if (!mbar_wait(&sm.full[st], ph, prm.timeout_ns, prm.status)) {
      failed = true;
      break;
    }
    const F64Box* Ab = sm.a[st];
    const F64Box* Bb = bi == bj ? sm.a[st] : sm.b[st];
#pragma unroll
    for (int ks = 0; ks < F64_KC / F64_KBOX; ++ks) {
      const double w0 = sm.w[st][ks * F64_KBOX + t], w1 = sm.w[st][ks * F64_KBOX + t + 4];
      // one 16-row slice of A at a time keeps the live set small
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        double ar[4], ai[4];
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = 32 * wi + 16 * mt + g + 8 * h;
            const double2 v = Ab[ks][r][(t + 4 * q) ^ (r & 7)];
            ar[2 * q + h] = v.x;
            ai[2 * q + h] = v.y;
          }
        // two column slices at a time: the two MMAs that share an accumulator are
        // three independent MMAs apart, hiding the DMMA latency
#pragma unroll
        for (int np = 0; np < 2; ++np) {
          double br[2][2], bim[2][2], bneg[2][2];
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int r = 32 * wj + 8 * (2 * np + h) + g;
              const double2 v = Bb[ks][r][(t + 4 * q) ^ (r & 7)];
              const double wq = q ? w1 : w0;
              br[h][q] = wq * v.x;
              bim[h][q] = wq * v.y;
              bneg[h][q] = -bim[h][q];
            }
          dmma_16x8x8(accR[mt][2 * np], ar, br[0]);
          dmma_16x8x8(accR[mt][2 * np + 1], ar, br[1]);
          dmma_16x8x8(accI[mt][2 * np], ai, br[0]);
          dmma_16x8x8(accI[mt][2 * np + 1], ai, br[1]);
          dmma_16x8x8(accR[mt][2 * np], ai, bim[0]);
          dmma_16x8x8(accR[mt][2 * np + 1], ai, bim[1]);
          dmma_16x8x8(accI[mt][2 * np], ar, bneg[0]);
          dmma_16x8x8(accI[mt][2 * np + 1], ar, bneg[1]);
        }
      }
    }
    // this warp is done with stage st
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.empty[st]);

    if (p0 + F64_KC >= prm.P) {
      // last slab of this item: add the tile into the packed upper triangle
      const int f = (int)(item / prm.ntile);
      double2* outf = prm.out + (int64_t)f * prm.npack;
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int i = bi * F64_B + 32 * wi + 16 * mt + g + 8 * (r >> 1);
            const int j = bj * F64_B + 32 * wj + 8 * nt + 2 * t + (r & 1);
            if (i <= j && j < prm.N) {
              double2* o = outf + (int64_t)j * (j + 1) / 2 + i;
              double2 v = *o;
              v.x += accR[mt][nt][r];
              v.y += accI[mt][nt][r];
              *o = v;
            }
          }
    }
  }
  if (failed && warp == 0 && lane == 0) {
    // never leave with copies still landing in this CTA's shared memory
    for (int64_t k = c; k < issued; ++k)
      mbar_drain(&sm.full[(int)(k % F64_ST)], (uint32_t)((k / F64_ST) & 1), prm.timeout_ns);
  }
}

// ---------------------------------------------------------------------------
// K1p: the product-first form of K1, for calls with several frequencies.
//
// The pair products z_p(i, j) = M(p, i) conj(M(p, j)) do not depend on the frequency:
// the reference forms them once and takes one ddot per frequency
// (src/susceptibility.f:1194-1205, :1779-1782). Per (p, i, j) that is 4 FP64 operations for
// z and 2 multiply-adds per frequency, against the 4 per frequency of K1, which
// folds the weight into one operand and contracts complex numbers. Here the
// contraction over p runs on DMMA with the products as the A operand (16 rows i of
// one column j, 8 pairs) and the weights as the B operand (8 pairs, 8 frequencies),
// re and im separately: 16 NT + 4 units for 8 NT frequencies instead of 32 NT
// (52 against 96 at 24 frequencies). Every thread forms exactly the products its
// fragment needs, in registers, so nothing is staged twice.
//
// Measured (1200 functions, 128000 pairs, 24 frequencies): 603 ms with K1, 295 ms here,
// 0.88 of the FP64 pipe at 1965 MHz for the 52 units; the error against 64-bit sums falls
// from 1.4e-14 to 1.0e-14 of the largest element.
//
// Bound: the FP64 pipe (DMMA and the products share it). A CTA of four warps owns
// 16 x 8 elements (two columns per warp) for one group of 8 NT frequencies, and streams
// 64-pair chunks of 16 + 8 columns of M and of the weights through F64P_ST TMA stages
// (SWIZZLE_128B). Long chunks matter more than resident warps: 16 pairs and three CTAs per
// SM 306 ms, 32 and three 299, 32 and two 297, 64 and two 295; four columns per warp spill.
//
// Work is dealt in whole tiles, one per CTA and round; the tiles of the last,
// partial round are cut along p into equal ranges, one per CTA, whose partial sums go
// to `part` and are added in CTA order by chi0_fp64p_reduce_kernel, so the result
// depends on the sizes only. Without `part` the last round stays whole.
constexpr int F64P_ST = 3;
constexpr int F64P_TI = 16;                              // tile rows of the polarisation
constexpr int F64P_MINPAIR = 256;                       // shortest p axis (pairs) worth cutting

// HW, the q -> 0 head and wings (src/susceptibility.f:1092-1157): the same sum for the rows
// i of [cprod | dcprod] against the three columns of dcprod. A warp owns 16 rows and all
// three columns, a CTA 64 rows; one more block of rows, dcprod itself, gives the head.
// Measured at 1100 columns, 48000 pairs, 24 frequencies: 0.64 ms with the cut tiles' sum,
// against 6.4 ms as a 72-row GEMM (weights folded into 3 x 24 rows, 64-row tiles).
//
// REAL, the -DINV build (src/susceptibility.f:1197): real M and chi, one product and one
// multiply-add per frequency: 1 + 8 NT units of the pipe, four columns per warp, 16 x 16 tiles.
// N = 1200, P = 10000, 24 frequencies: 19.4 ms on K1r, 11.2 here (0.90 of the FP64 pipe); K1r
// keeps the shapes that f64_on_k1 gives it.
constexpr int F64P_CPLX = 0, F64P_HW = 1, F64P_REAL = 2;   // MODE
template <int MODE>
struct F64PTile {
  static constexpr bool HW = MODE == F64P_HW, REAL = MODE == F64P_REAL;
  static constexpr int TI = HW ? 64 : F64P_TI;
  static constexpr int JW = HW ? 3 : (REAL ? 4 : 2);           // columns per warp
  static constexpr int TJ = HW ? 8 : 4 * JW;                   // columns of a box of j
  static constexpr int CTAS = 2;                               // resident CTAs per SM
  static constexpr int KC = HW ? 16 : 64;                      // band pairs per stage
  static constexpr int NBOX = KC / (REAL ? 16 : F64_KBOX);     // 128-byte boxes per stage
  static constexpr int ELEMS = JW * 4 * F64_THREADS;           // of a CTA, per 8 frequencies
};

template <int NT, int MODE>
struct __align__(1024) F64PSmem {
  static constexpr int KC = F64PTile<MODE>::KC;
  double2 a[F64P_ST][F64PTile<MODE>::NBOX][F64PTile<MODE>::TI][F64_KBOX];
  double2 b[F64P_ST][F64PTile<MODE>::NBOX][F64PTile<MODE>::TJ][F64_KBOX];
  double w[F64P_ST][KC / 16][8 * NT][16];   // row f's 16-byte chunk c stored at c ^ (f & 7)
  uint64_t full[F64P_ST];
  uint64_t empty[F64P_ST];
};

struct F64PParams {
  int N, nw, f0;           // matrix size, frequencies of the call, first frequency of this launch
  int ntile, nchunk;
  int64_t items;           // ntile x frequency groups
  int64_t whole;           // items dealt whole: rounds x grid (all of them without `part`)
  double2* out;            // packed polarisation (REAL: as doubles); HW: wing (3, N, nw)
  double2* head;           // HW: head (6, nw)
  int64_t npack;
  double2* part;           // [CTA][2 slots][elements] partial tiles (REAL: doubles), or NULL
  int* status;
  uint64_t timeout_ns;
};

// The segments of one CTA: whole items blockIdx.x, + gridDim.x, ... below `whole`, then
// its share [u, u1) of the remaining items' chunks, cut at item boundaries.
struct F64PSeg {
  int64_t item;   // next whole item
  int64_t u, u1;
  int nseg;       // partial-range segments handed out
  __device__ __forceinline__ void init(const F64PParams& p, int cta, int grid) {
    item = cta;
    const int64_t tail = (p.items - p.whole) * (int64_t)p.nchunk;
    u = tail * cta / grid;
    u1 = tail * (cta + 1) / grid;
    nseg = 0;
  }
  // Next segment: item, chunks [k0, k1), slot (-1: a whole item). False at the end.
  __device__ __forceinline__ bool next(const F64PParams& p, int grid, int64_t* it, int* k0, int* k1, int* slot) {
    if (item < p.whole) {
      *it = item;
      *k0 = 0;
      *k1 = p.nchunk;
      *slot = -1;
      item += grid;
      return true;
    }
    if (u >= u1) return false;
    const int64_t t = u / p.nchunk;
    *it = p.whole + t;
    *k0 = (int)(u - t * p.nchunk);
    const int64_t e = min(u1, (t + 1) * (int64_t)p.nchunk);
    *k1 = (int)(e - t * p.nchunk);
    *slot = (*k0 == 0 && *k1 == p.nchunk) ? -1 : min(nseg, 1);
    ++nseg;
    u = e;
    return true;
  }
};

// Tile t of the upper triangle in 16-row x 8-column blocks: column block bj has
// bj / 2 + 1 row blocks, so blocks 2m and 2m + 1 start at m (m + 1) and (m + 1)^2.
__host__ __device__ __forceinline__ void f64p_decode(int t, int* bi, int* bj) {
  int m = (int)((sqrtf(4.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while (m * (m + 1) > t) --m;
  while ((m + 1) * (m + 2) <= t) ++m;
  const int r = t - m * (m + 1);
  *bj = 2 * m + (r > m ? 1 : 0);
  *bi = r > m ? r - (m + 1) : r;
}
template <int MODE>
__device__ __forceinline__ void f64p_tile(int t, int* bi, int* bj) {
  if constexpr (MODE == F64P_REAL) decode_tile(t, bi, bj);
  else f64p_decode(t, bi, bj);
}
template <int MODE>
static int f64p_tiles(int N) {
  const int nbj = (N + F64PTile<MODE>::TJ - 1) / F64PTile<MODE>::TJ, m = nbj / 2;
  return MODE == F64P_REAL ? nbj * (nbj + 1) / 2 : m * (m + 1) + (nbj & 1) * (m + 1);
}

template <int NT, int MODE>
struct F64PAcc {
  double re[F64PTile<MODE>::JW][NT][4], im[F64PTile<MODE>::JW][NT][4];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int jj = 0; jj < F64PTile<MODE>::JW; ++jj)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int r = 0; r < 4; ++r) re[jj][nt][r] = im[jj][nt][r] = 0.0;
  }
  static constexpr int ELEMS = NT * F64PTile<MODE>::ELEMS;   // of a CTA
};

// Adds a tile held as accumulator fragments (row g + 8 (r / 2), frequency
// 8 nt + 2 t + (r & 1)) into the output.
template <int NT, int MODE>
__device__ __forceinline__ void f64p_store(const F64PParams& prm, int64_t item, const F64PAcc<NT, MODE>& acc) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int fb = prm.f0 + (int)(item / prm.ntile) * 8 * NT;
  if constexpr (MODE == F64P_HW) {
    const int bi = (int)(item % prm.ntile);
    const bool hd = bi == prm.ntile - 1;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int row = 16 * warp + g + 8 * (r >> 1), f = fb + 8 * nt + 2 * t + (r & 1);
        const int i = hd ? row : bi * F64PTile<MODE>::TI + row;
        if (f >= prm.nw || i >= (hd ? 3 : prm.N)) continue;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (hd && i > a) continue;
          double2* o = hd ? prm.head + a * (a + 1) / 2 + i + 6 * (int64_t)f
                          : prm.out + a + 3 * ((int64_t)i + (int64_t)prm.N * f);
          double2 v = *o;
          v.x += acc.re[a][nt][r];
          v.y += acc.im[a][nt][r];
          *o = v;
        }
      }
    return;
  }
  int bi, bj;
  f64p_tile<MODE>((int)(item % prm.ntile), &bi, &bj);
#pragma unroll
  for (int jj = 0; jj < F64PTile<MODE>::JW; ++jj) {
    const int j = bj * F64PTile<MODE>::TJ + F64PTile<MODE>::JW * warp + jj;
    if (j >= prm.N) continue;
    double2* oj = prm.out + (int64_t)j * (j + 1) / 2;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int i = bi * F64P_TI + g + 8 * (r >> 1), f = fb + 8 * nt + 2 * t + (r & 1);
        if (i > j || f >= prm.nw) continue;
        if constexpr (MODE == F64P_REAL) {
          reinterpret_cast<double*>(prm.out)[(int64_t)j * (j + 1) / 2 + (int64_t)f * prm.npack + i] += acc.re[jj][nt][r];
          continue;
        }
        double2* o = oj + (int64_t)f * prm.npack + i;
        double2 v = *o;
        v.x += acc.re[jj][nt][r];
        v.y += acc.im[jj][nt][r];
        *o = v;
      }
  }
}

// mapI: boxes of the rows i; mapJ: the 8-column boxes of j; mapH (HW): dcprod as rows
template <int NT, int MODE>
__global__ void __launch_bounds__(F64_THREADS, F64PTile<MODE>::CTAS)
    chi0_fp64p_kernel(const __grid_constant__ CUtensorMap mapI, const __grid_constant__ CUtensorMap mapJ,
                      const __grid_constant__ CUtensorMap mapW, const __grid_constant__ CUtensorMap mapH,
                      F64PParams prm) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  using Smem = F64PSmem<NT, MODE>;
  constexpr bool HW = F64PTile<MODE>::HW, REAL = F64PTile<MODE>::REAL;
  constexpr int JW = F64PTile<MODE>::JW, KC = F64PTile<MODE>::KC;
  Smem& sm = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  if (threadIdx.x == 0) {
    for (int s = 0; s < F64P_ST; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], F64_WARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();

  // warp 0, lane 0 issues the copies, F64P_ST - 2 chunks ahead of the chunk it computes: a
  // stage is refilled a whole chunk after it was read, so the issuer rarely waits
  F64PSeg ps;
  int64_t p_item = 0;
  int pk = 0, pk1 = 0, p_slot, py = 0, pyj = 0, pf = 0;
  bool p_more = false, p_head = false;
  uint32_t issued = 0;
  auto enter = [&] {
    if constexpr (HW) {
      const int bi = (int)(p_item % prm.ntile);
      p_head = bi == prm.ntile - 1;
      py = p_head ? 0 : bi * F64PTile<MODE>::TI;
    } else {
      int bi, bj;
      f64p_tile<MODE>((int)(p_item % prm.ntile), &bi, &bj);
      py = bi * F64P_TI;
      pyj = bj * F64PTile<MODE>::TJ;
    }
    pf = prm.f0 + (int)(p_item / prm.ntile) * 8 * NT;
  };
  auto issue = [&] {
    const int st = (int)(issued % F64P_ST);
    mbar_arrive_expect_tx(&sm.full[st], (uint32_t)(sizeof(sm.a[0]) + sizeof(sm.b[0]) + sizeof(sm.w[0])));
    const int x = pk * KC * (REAL ? 1 : 2);   // in doubles; a box holds 16
#pragma unroll
    for (int h = 0; h < F64PTile<MODE>::NBOX; ++h) {
      tma_load_2d(&sm.a[st][h][0][0], HW && p_head ? &mapH : &mapI, x + 16 * h, py, &sm.full[st]);
      tma_load_2d(&sm.b[st][h][0][0], &mapJ, x + 16 * h, pyj, &sm.full[st]);
    }
#pragma unroll
    for (int h = 0; h < KC / 16; ++h) tma_load_2d(&sm.w[st][h][0][0], &mapW, pk * KC + 16 * h, pf, &sm.full[st]);
    ++issued;
    if (++pk == pk1) {
      p_more = ps.next(prm, gridDim.x, &p_item, &pk, &pk1, &p_slot);
      if (p_more) enter();
    }
  };
  if (threadIdx.x == 0) {
    ps.init(prm, blockIdx.x, gridDim.x);
    p_more = ps.next(prm, gridDim.x, &p_item, &pk, &pk1, &p_slot);
    if (p_more) enter();
    while (p_more && issued < F64P_ST - 2) issue();
  }

  F64PSeg seg;
  seg.init(prm, blockIdx.x, gridDim.x);
  int64_t item;
  int k0, k1, slot;
  uint32_t c = 0;   // chunks computed
  bool ok = true;
  while (ok && seg.next(prm, gridDim.x, &item, &k0, &k1, &slot)) {
    F64PAcc<NT, MODE> acc;
    acc.zero();
    for (int k = k0; k < k1; ++k, ++c) {
      const int st = (int)(c % F64P_ST);
      if (warp == 0) {
        int good = 1;
        if (lane == 0 && p_more) {
          // the next chunk to issue is c + F64P_ST - 2, into the stage of chunk c - 2
          if (c >= 2)
            good = mbar_wait(&sm.empty[(c - 2) % F64P_ST], ((c - 2) / F64P_ST) & 1u, prm.timeout_ns, prm.status);
          if (good) issue();
        }
        if (!__shfl_sync(0xffffffffu, good, 0)) {
          ok = false;
          break;
        }
      }
      if (!mbar_wait(&sm.full[st], (c / F64P_ST) & 1u, prm.timeout_ns, prm.status)) {
        ok = false;
        break;
      }
#pragma unroll
      for (int ks = 0; ks < KC / F64_KBOX; ++ks) {
        double wf[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int p = F64_KBOX * (ks & 1) + t + 4 * q;
            wf[nt][q] = sm.w[st][ks >> 1][8 * nt + g][(((p >> 1) ^ g) << 1) | (p & 1)];
          }
        if constexpr (REAL) {
          // pair k of row r sits in 16-byte chunk (k / 2) ^ (r & 7) of its box
          auto at = [&](const double2 (*box)[F64_KBOX], int r, int q) {
            const int p = F64_KBOX * (ks & 1) + t + 4 * q;
            return reinterpret_cast<const double*>(box[r])[(((p >> 1) ^ (r & 7)) << 1) | (p & 1)];
          };
          double ar[4];
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h) ar[2 * q + h] = at(sm.a[st][ks >> 1], g + 8 * h, q);
#pragma unroll
          for (int jj = 0; jj < JW; ++jj) {
            const double b[2] = {at(sm.b[st][ks >> 1], JW * warp + jj, 0), at(sm.b[st][ks >> 1], JW * warp + jj, 1)};
            const double z[4] = {ar[0] * b[0], ar[1] * b[0], ar[2] * b[1], ar[3] * b[1]};
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) dmma_16x8x8(acc.re[jj][nt], z, wf[nt]);
          }
        } else {
          double2 a[4];   // a[2q + h] = M(pair t + 4q, row g + 8h)
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              a[2 * q + h] = sm.a[st][ks][(HW ? 16 * warp : 0) + g + 8 * h][(t + 4 * q) ^ g];
#pragma unroll
          for (int jj = 0; jj < JW; ++jj) {
            const int rj = HW ? jj : JW * warp + jj;
            const double2 b0 = sm.b[st][ks][rj][t ^ (rj & 7)];
            const double2 b1 = sm.b[st][ks][rj][(t + 4) ^ (rj & 7)];
            double z[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const double2 b = e < 2 ? b0 : b1;
              z[e] = fma(a[e].x, b.x, a[e].y * b.y);
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) dmma_16x8x8(acc.re[jj][nt], z, wf[nt]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const double2 b = e < 2 ? b0 : b1;
              z[e] = fma(a[e].y, b.x, -(a[e].x * b.y));
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) dmma_16x8x8(acc.im[jj][nt], z, wf[nt]);
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.empty[st]);
    }
    if (!ok) break;
    if (slot < 0) {
      f64p_store<NT, MODE>(prm, item, acc);
    } else {
      const int64_t at = ((int64_t)blockIdx.x * 2 + slot) * F64PAcc<NT, MODE>::ELEMS + threadIdx.x;
#pragma unroll
      for (int jj = 0; jj < JW; ++jj)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int r = 0; r < 4; ++r)
            if constexpr (REAL)
              reinterpret_cast<double*>(prm.part)[at + ((jj * NT + nt) * 4 + r) * F64_THREADS] = acc.re[jj][nt][r];
            else
              prm.part[at + ((jj * NT + nt) * 4 + r) * F64_THREADS] = make_double2(acc.re[jj][nt][r], acc.im[jj][nt][r]);
    }
  }
  if (!ok && threadIdx.x == 0) {
    // never leave with copies still landing in this CTA's shared memory
    for (uint32_t k = c; k < issued; ++k)
      mbar_drain(&sm.full[k % F64P_ST], (k / F64P_ST) & 1u, prm.timeout_ns);
  }
}

// One CTA per boundary b between the ranges of CTAs b and b + 1 of the accumulation
// (grid `ncta`): when it falls inside an item and is the first to do so, adds the item's
// partial tiles in CTA order into the output.
template <int NT, int MODE>
__global__ void __launch_bounds__(F64_THREADS) chi0_fp64p_reduce_kernel(F64PParams prm, int ncta) {
  const int64_t tail = (prm.items - prm.whole) * (int64_t)prm.nchunk;
  const int c = blockIdx.x + 1;
  const int64_t u = tail * c / ncta;
  const int64_t t = u / prm.nchunk;
  const int64_t t0 = t * prm.nchunk, t1 = t0 + prm.nchunk;
  if (u == t0 || u >= tail) return;
  const int64_t up = tail * (c - 1) / ncta;
  if (up > t0) return;   // an earlier boundary already lies inside this item
  F64PAcc<NT, MODE> acc;
  acc.zero();
  for (int k = c - 1; k < ncta; ++k) {
    const int64_t s = tail * k / ncta;
    if (s >= t1) break;
    if (tail * (k + 1) / ncta == s) continue;   // an empty range
    // the item is a CTA's first segment when its range starts inside it
    const int slot = s >= t0 ? 0 : 1;
    const int64_t at = ((int64_t)k * 2 + slot) * F64PAcc<NT, MODE>::ELEMS + threadIdx.x;
#pragma unroll
    for (int jj = 0; jj < F64PTile<MODE>::JW; ++jj)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int64_t x = at + ((jj * NT + nt) * 4 + r) * F64_THREADS;
          if constexpr (MODE == F64P_REAL) {
            acc.re[jj][nt][r] += reinterpret_cast<const double*>(prm.part)[x];
            continue;
          }
          const double2 v = prm.part[x];
          acc.re[jj][nt][r] += v.x;
          acc.im[jj][nt][r] += v.y;
        }
  }
  f64p_store<NT, MODE>(prm, prm.whole + t, acc);
}

// Tensor map of M as a 2-D FP64 array: pairs (re, im interleaved) contiguous,
// columns ldc complex apart; boxes of 8 pairs x `cols` columns, SWIZZLE_128B. real: M holds
// doubles, 16 pairs a box.
static int f64_map(CUtensorMap* map, const double2* M, int64_t ldc, int64_t P, int N, int cols,
                   bool real = false) {
  const uint64_t dims[2] = {(uint64_t)((real ? 1 : 2) * P), (uint64_t)N};
  const uint64_t strides[1] = {(uint64_t)ldc * (real ? 8 : 16)};
  const uint32_t box[2] = {2 * F64_KBOX, (uint32_t)cols};
  return encode_tmap(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, M, dims, strides, box,
                     CU_TENSOR_MAP_SWIZZLE_128B);
}

// What both launchers share.
struct F64Call {
  int num_sms;
  const double2* M;
  int64_t ldc, P;
  int N;
  const double* W;
  int64_t ldw;
  int nw;
  double2* out;
  double2* part;
  size_t part_bytes;
  int* status;
  uint64_t timeout_ns;
  cudaStream_t stream;
};

// K1 for the `n` frequencies from f0.
static int f64_launch(const F64Call& q, int f0, int n, int* launches) {
  const int nblk = (q.N + F64_B - 1) / F64_B;
  F64Params prm;
  prm.P = q.P;
  prm.N = q.N;
  prm.W = q.W + (int64_t)f0 * q.ldw;
  prm.ldw = q.ldw;
  prm.nw = n;
  prm.npack = (int64_t)q.N * (q.N + 1) / 2;
  prm.out = q.out + (int64_t)f0 * prm.npack;
  prm.ntile = nblk * (nblk + 1) / 2;
  prm.nitems = (int64_t)prm.ntile * n;
  prm.status = q.status;
  prm.timeout_ns = q.timeout_ns;
  CUtensorMap map;
  const int e = f64_map(&map, q.M, q.ldc, q.P, q.N, F64_B);
  if (e) return e;
  const size_t smem = sizeof(F64Smem) + 1024;
  if (cudaFuncSetAttribute(chi0_fp64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return -2;
  const int grid = (int)std::min<int64_t>(prm.nitems, (int64_t)2 * q.num_sms);
  chi0_fp64_kernel<<<grid, F64_THREADS, smem, q.stream>>>(map, prm);
  ++*launches;
  return 0;
}

template <int MODE>
static size_t f64p_part_bytes(int num_sms, int nt) {
  return (MODE == F64P_REAL ? sizeof(double) : sizeof(double2)) * (size_t)F64PTile<MODE>::CTAS * num_sms * 2 * nt *
         F64PTile<MODE>::ELEMS;
}

// The head and wings' second operand and outputs (HW): dcprod (ldd, 3) and head.
struct F64Head {
  const double2* dc;
  int64_t ldd;
  double2* head;
};

// K1p for `groups` groups of 8 NT frequencies from f0 (the last may be ragged).
template <int NT, int MODE>
static int f64p_launch(const F64Call& q, const F64Head& hw, int f0, int groups, int* launches) {
  using Tile = F64PTile<MODE>;
  constexpr bool HW = Tile::HW, REAL = Tile::REAL;
  F64PParams prm;
  prm.N = q.N;
  prm.nw = q.nw;
  prm.f0 = f0;
  prm.ntile = HW ? (q.N + Tile::TI - 1) / Tile::TI + 1 : f64p_tiles<MODE>(q.N);
  const int64_t nchunk = (q.P + Tile::KC - 1) / Tile::KC;
  if (nchunk > 0x7fffffff / (2 * Tile::KC)) return -3;   // pair coordinates are 32-bit
  prm.nchunk = (int)nchunk;
  prm.items = (int64_t)prm.ntile * groups;
  prm.out = q.out;
  prm.head = hw.head;
  prm.npack = (int64_t)q.N * (q.N + 1) / 2;
  prm.status = q.status;
  prm.timeout_ns = q.timeout_ns;
  const int64_t slots = (int64_t)Tile::CTAS * q.num_sms;
  const bool cut = q.part && q.part_bytes >= f64p_part_bytes<MODE>(q.num_sms, NT) &&
                   q.P >= F64P_MINPAIR && prm.items % slots != 0;
  // fewer items than slots: as many CTAs as get half of the shortest cut axis each
  const int64_t fit = cut ? std::max(prm.items, prm.items * prm.nchunk / (F64P_MINPAIR / 2 / Tile::KC)) : prm.items;
  const int grid = (int)std::min(slots, fit);
  prm.whole = cut ? prm.items / grid * grid : prm.items;
  prm.part = cut ? q.part : nullptr;
  CUtensorMap mi, mj, mw, mh;
  int e;
  if (HW) {
    e = f64_map(&mj, hw.dc, hw.ldd, q.P, 3, Tile::TJ);
    if (!e) e = f64_map(&mh, hw.dc, hw.ldd, q.P, 3, Tile::TI);
    if (!e && q.N > 0) e = f64_map(&mi, q.M, q.ldc, q.P, q.N, Tile::TI);
    if (q.N == 0) mi = mh;
  } else {
    e = f64_map(&mi, q.M, q.ldc, q.P, q.N, Tile::TI, REAL);
    if (!e) e = f64_map(&mj, q.M, q.ldc, q.P, q.N, Tile::TJ, REAL);
    mh = mi;
  }
  if (!e) {
    // pairs past the end of the weights read as zeros
    const uint64_t dims[2] = {(uint64_t)q.P, (uint64_t)q.nw};
    const uint64_t strides[1] = {(uint64_t)q.ldw * 8};
    const uint32_t box[2] = {16, 8 * NT};
    e = encode_tmap(&mw, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, q.W, dims, strides, box,
                    CU_TENSOR_MAP_SWIZZLE_128B);
  }
  if (e) return e;
  const size_t smem = sizeof(F64PSmem<NT, MODE>) + 1024;
  if (cudaFuncSetAttribute(chi0_fp64p_kernel<NT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return -2;
  chi0_fp64p_kernel<NT, MODE><<<grid, F64_THREADS, smem, q.stream>>>(mi, mj, mw, mh, prm);
  ++*launches;
  if (prm.whole < prm.items && grid > 1) {
    chi0_fp64p_reduce_kernel<NT, MODE><<<grid - 1, F64_THREADS, 0, q.stream>>>(prm, grid);
    ++*launches;
  }
  return 0;
}

// Which frequencies of a call go to K1 (K1r): times in us of the two forms, from a fit to both
// over 14 widths from 17 to 1500, 1 to 12800 pairs and 1 to 48 frequencies. K1 works on whole
// 64 x 64 tiles of one frequency, two at once per SM, 4 (real: 1) units an element and pair,
// with pairs padded to 16; K1p on 16 x 8 (16 x 16) tiles of eight frequencies a block, 4 + 16 a
// block (1 + 8), with pairs padded to 64 unless the last round is cut. So K1 is better for few
// frequencies of a wide matrix, and for few pairs, which leave K1p's padding and its longer
// epilogue. `call`, `round`: start, and a round of resident tiles; `unit`: against the pipe's 64
// multiply-adds per clock and SM at 1.9 GHz (below and from F64P_MINPAIR pairs); `alone`: a tile
// without a second one on its SM, of half of two; `cut`: partial tiles and their sum. us, K1 /
// K1p (N, P, frequencies): complex 65, 80, 36: 36 / 44; 640, 16, 12: 57 / 74; 900, 80, 5:
// 99 / 118; 1500, 16, 36: 889 / 1108; 900, 12800, 3: 6777 / 7576; 1500, 12800, 4: 18349 / 20767;
// the other way round 150, 80, 48: 45 / 34; 640, 80, 24: 185 / 149; 1500, 80, 48: 2050 / 1714;
// 400, 12800, 4: 2866 / 1567. Real 65, 80, 48: 26 / 36; 900, 16, 36: 228 / 309; 1500, 80, 36: 910 / 1033;
// 1500, 12800, 4: 7643 / 9060; the other way round 300, 80, 24: 50 / 41; 300, 10000, 24: 2395 /
// 781; 1200, 10000, 5: 4783 / 4564. Of 3807 shapes of each from 65 columns on, 41 (complex) and 78
// (real) take over 3 % more than the better form.
struct F64Cost {
  double k1_call, k1_round, k1_unit, k1_alone;
  double p_call, p_round, p_block, p_unit, p_unit_long, p_alone, p_cut;
};
template <int MODE>
static double f64_us_k1(int sms, int N, int64_t P, int n, const F64Cost& c) {
  const int64_t nblk = (N + F64_B - 1) / F64_B, per_sm = (nblk * (nblk + 1) / 2 * n + sms - 1) / sms;
  const double tile = (MODE == F64P_REAL ? 1 : 4) * F64_B * F64_B * (double)align_up((size_t)P, 16) / (64 * 1900.0);
  return c.k1_call + c.k1_round * (double)((per_sm + 1) / 2) +
         c.k1_unit * tile * ((double)(per_sm / 2) * 2 + (double)(per_sm % 2) * c.k1_alone);
}
template <int MODE>
static double f64_us_k1p(int sms, bool part, int N, int64_t P, int nt, int groups, const F64Cost& c) {
  using Tile = F64PTile<MODE>;
  const int64_t items = (int64_t)f64p_tiles<MODE>(N) * groups, per_sm = (items + sms - 1) / sms;
  const double pair = (MODE == F64P_REAL ? 1 + 8.0 * nt : 4 + 16.0 * nt) * F64P_TI * Tile::TJ / (64 * 1900.0);
  double us = c.p_call + (double)((per_sm + 1) / 2) * (c.p_round + c.p_block * nt);
  if (part && P >= F64P_MINPAIR && items % (2 * sms) != 0)
    return us + c.p_cut + c.p_unit_long * pair * (double)P * (double)items / sms;
  return us + (P < F64P_MINPAIR ? c.p_unit : c.p_unit_long) * pair * (double)align_up((size_t)P, Tile::KC) *
                  ((double)(per_sm / 2) * 2 + (double)(per_sm % 2) * c.p_alone);
}
// Frequencies of a call on K1, the last ones: all nw, the remainder of the groups of 24, or none.
template <int MODE>
static int f64_on_k1(int sms, bool part, int N, int64_t P, int nw) {
  constexpr F64Cost c = MODE == F64P_REAL
                            ? F64Cost{7.1, 11.7, 1.93, 1.8, 6.8, 1.0, 6.1, 0.91, 1.15, 1.53, 11.9}
                            : F64Cost{6.5, 13.7, 1.17, 1.41, 6.9, 1.8, 2.5, 1.10, 1.19, 1.24, 13.3};
  const int r = nw % 24 > 16 ? 0 : nw % 24, full = (nw - r + 23) / 24;
  double us = full ? f64_us_k1p<MODE>(sms, part, N, P, 3, full, c) : 0.0;
  int n = 0;
  if (r > 0) {
    const double k1 = f64_us_k1<MODE>(sms, N, P, r, c), k1p = f64_us_k1p<MODE>(sms, part, N, P, r > 8 ? 2 : 1, 1, c);
    if (k1 <= k1p) n = r;
    us += std::min(k1, k1p);
  }
  return f64_us_k1<MODE>(sms, N, P, nw, c) <= us ? nw : n;
}
int fp64_on_k1(bool real, int sms, bool part, int N, int64_t P, int nw) {
  return real ? f64_on_k1<F64P_REAL>(sms, part, N, P, nw) : f64_on_k1<F64P_CPLX>(sms, part, N, P, nw);
}

static int f64r_launch(const F64Call& q, int f0, int n, int* launches);

// Frequencies go to K1p in groups of 24 (three DMMA column blocks) and a remainder in the
// narrowest form that holds it, unless they go to K1 (K1r).
template <int MODE>
static int f64_run(const F64Call& q, int* launches) {
  const int n1 = fp64_on_k1(MODE == F64P_REAL, q.num_sms, q.part != nullptr, q.N, q.P, q.nw), rest = q.nw - n1;
  int full = rest / 24, r = rest % 24, e = 0;
  if (r > 16) ++full, r = 0;
  if (full) e = f64p_launch<3, MODE>(q, {}, 0, full, launches);
  if (!e && r > 8) e = f64p_launch<2, MODE>(q, {}, 24 * full, 1, launches);
  else if (!e && r > 0) e = f64p_launch<1, MODE>(q, {}, 24 * full, 1, launches);
  if (!e && n1 > 0) e = MODE == F64P_REAL ? f64r_launch(q, rest, n1, launches) : f64_launch(q, rest, n1, launches);
  return e;
}

// Bytes that hold the partial tiles of any call.
size_t fp64_part_bytes(int num_sms) {
  return std::max({f64p_part_bytes<F64P_CPLX>(num_sms, 3), f64p_part_bytes<F64P_HW>(num_sms, 3),
                   f64p_part_bytes<F64P_REAL>(num_sms, 3)});
}

// Enqueues the FP64 accumulation over one slab of band pairs. W holds the weights of
// exactly these pairs (leading dimension ldw, a multiple of 16, padding zeroed, 16-byte
// aligned).
int launch_chi0_fp64(spx_ctx* ctx, const double2* M, int64_t ldc, int64_t P, int N,
                     const double* W, int64_t ldw, int nw, double2* out, cudaStream_t stream,
                     int* launches) {
  if (P <= 0 || N <= 0 || nw <= 0) return SPX_OK;
  const uint64_t timeout_ns =
      (uint64_t)(ctx->opt.timeout_ms > 0 ? ctx->opt.timeout_ms : 4000) * 1000000ull;
  const F64Call q{ctx->num_sms, M, ldc, P, N, W, ldw, nw, out, (double2*)ctx->part, ctx->part_bytes,
                  ctx->d_status, timeout_ns, stream};
  const int e = f64_run<F64P_CPLX>(q, launches);
  if (e) return set_error(ctx, SPX_ECUDA, "chi0_fp64 kernels: tensor map or attribute failed (" +
                                              std::to_string(e) + ")");
  return check_cuda(ctx, cudaGetLastError(), "chi0_fp64 kernel launch");
}

// head(:, f) += sum_p dc(p, k1) conj(dc(p, k2)) w(p, f), wing(k2, i, f) += sum_p M(p, i)
// conj(dc(p, k2)) w(p, f): M (ldc, dim), dc (ldd, 3), W (ldw, nw) with ldw even and W 16-byte
// aligned. P < 2^30.
int launch_headwings(spx_ctx* ctx, const double2* M, int64_t ldc, int64_t P, int dim,
                     const double2* dc, int64_t ldd, const double* W, int64_t ldw, int nw,
                     double2* head, double2* wing, cudaStream_t stream) {
  if (P <= 0 || nw <= 0) return SPX_OK;
  const uint64_t timeout_ns =
      (uint64_t)(ctx->opt.timeout_ms > 0 ? ctx->opt.timeout_ms : 4000) * 1000000ull;
  const F64Call q{ctx->num_sms, M, ldc, P, dim, W, ldw, nw, wing, (double2*)ctx->part, ctx->part_bytes,
                  ctx->d_status, timeout_ns, stream};
  const F64Head hw{dc, ldd, head};
  int full = nw / 24, r = nw % 24, e = 0, launches = 0;
  if (r > 16) ++full, r = 0;
  if (full) e = f64p_launch<3, F64P_HW>(q, hw, 0, full, &launches);
  if (!e && r > 8) e = f64p_launch<2, F64P_HW>(q, hw, 24 * full, 1, &launches);
  else if (!e && r > 0) e = f64p_launch<1, F64P_HW>(q, hw, 24 * full, 1, &launches);
  if (e) return set_error(ctx, SPX_ECUDA, "head and wings: tensor map or attribute failed (" +
                                              std::to_string(e) + ")");
  return check_cuda(ctx, cudaGetLastError(), "head and wings launch");
}

// launch_chi0_fp64 with explicit device resources instead of a context: used by the
// allocation-free entry point, whose status word and weights live in static
// device memory.
int launch_chi0_fp64_noctx(int num_sms, int* status, uint64_t timeout_ns, const double2* M,
                           int64_t ldc, int64_t P, int N, const double* W, int64_t ldw, int nw,
                           double2* out, cudaStream_t stream) {
  if (P <= 0 || N <= 0 || nw <= 0) return SPX_OK;
  const F64Call q{num_sms, M, ldc, P, N, W, ldw, nw, out, nullptr, 0, status, timeout_ns, stream};
  int launches = 0;
  if (f64_run<F64P_CPLX>(q, &launches)) return SPX_ECUDA;
  return cudaGetLastError() == cudaSuccess ? SPX_OK : SPX_ECUDA;
}

// ---------------------------------------------------------------------------
// K1r: the -DINV build for few frequencies (MCOMPLEX_dp = real_dp, src/cppmacro.h:53-64), where
// re(k) = cprod(k,i) * cprod(k,j) (src/susceptibility.f:1197) and chi is real:
//   chi_f(i, j) += sum_p M(p, i) M(p, j) w(p, f),  i <= j,
// on the same pipeline as K1 with one 2-D TMA box of 16 pairs x 64 columns per
// panel and stage (128-byte rows, SWIZZLE_128B: pair k of row r sits in 16-byte
// chunk (k/2) ^ (r & 7)), and one DMMA per 8 x 8 real product.
typedef double F64RBox[F64_B][F64_KC];

struct __align__(1024) F64RSmem {
  F64RBox a[F64_ST];
  F64RBox b[F64_ST];
  double w[F64_ST][F64_KC];
  uint64_t full[F64_ST];
  uint64_t empty[F64_ST];
};

__device__ __forceinline__ double f64r_at(const F64RBox& box, int r, int k) {
  return box[r][(((k >> 1) ^ (r & 7)) << 1) | (k & 1)];
}

__global__ void __launch_bounds__(F64_THREADS, 2)
    chi0_fp64_real_kernel(const __grid_constant__ CUtensorMap mapM, F64Params prm, double* outr) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  F64RSmem& sm = *reinterpret_cast<F64RSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                              ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < F64_ST; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], F64_WARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();
  const int64_t nchunk = (prm.P + F64_KC - 1) / F64_KC;
  const int64_t my_items = prm.nitems > blockIdx.x
                               ? (prm.nitems - blockIdx.x + gridDim.x - 1) / gridDim.x
                               : 0;
  const int64_t total = my_items * nchunk;
  auto chunk_item = [&](int64_t c) { return blockIdx.x + (c / nchunk) * (int64_t)gridDim.x; };
  auto chunk_p0 = [&](int64_t c) { return (c % nchunk) * (int64_t)F64_KC; };
  auto issue = [&](int64_t c) {
    const int st = (int)(c % F64_ST);
    const int64_t item = chunk_item(c), p0 = chunk_p0(c);
    const int f = (int)(item / prm.ntile);
    int bi, bj;
    decode_tile((int)(item % prm.ntile), &bi, &bj);
    const bool same = bi == bj;
    mbar_arrive_expect_tx(&sm.full[st], (uint32_t)((same ? 1 : 2) * sizeof(F64RBox) + F64_KC * 8));
    tma_load_2d(&sm.a[st][0][0], &mapM, (int)p0, bi * F64_B, &sm.full[st]);
    if (!same) tma_load_2d(&sm.b[st][0][0], &mapM, (int)p0, bj * F64_B, &sm.full[st]);
    bulk_g2s(&sm.w[st][0], prm.W + (int64_t)f * prm.ldw + p0, F64_KC * 8, &sm.full[st]);
  };
  int64_t issued = total < F64_ST - 1 ? total : (int64_t)(F64_ST - 1);
  if (warp == 0 && lane == 0)
    for (int64_t c = 0; c < issued; ++c) issue(c);

  const int wi = warp & 1, wj = warp >> 1;
  const int g = lane >> 2, t = lane & 3;
  double acc[2][4][4];
  bool failed = false;
  int64_t c = 0;
  for (; c < total; ++c) {
    const int st = (int)(c % F64_ST);
    const uint32_t ph = (uint32_t)((c / F64_ST) & 1);
    const int64_t item = chunk_item(c), p0 = chunk_p0(c);
    int bi, bj;
    decode_tile((int)(item % prm.ntile), &bi, &bj);
    if (p0 == 0) {
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int r = 0; r < 4; ++r) acc[mt][nt][r] = 0.0;
    }
    if (warp == 0 && c + F64_ST - 1 < total) {
      const int64_t prev = c - 1;
      int ok = 1;
      if (lane == 0) {
        if (prev >= 0)
          ok = mbar_wait(&sm.empty[(int)(prev % F64_ST)], (uint32_t)((prev / F64_ST) & 1),
                         prm.timeout_ns, prm.status);
        if (ok) issue(c + F64_ST - 1);
      }
      if (!__shfl_sync(0xffffffffu, ok, 0)) {
        failed = true;
        break;
      }
      issued = c + F64_ST;
    }
    if (!mbar_wait(&sm.full[st], ph, prm.timeout_ns, prm.status)) {
      failed = true;
      break;
    }
    const F64RBox& A = sm.a[st];
    const F64RBox& B = bi == bj ? sm.a[st] : sm.b[st];
#pragma unroll
    for (int ks = 0; ks < F64_KC / 8; ++ks) {
      const double w0 = sm.w[st][8 * ks + t], w1 = sm.w[st][8 * ks + t + 4];
      double bq[4][2];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int r = 32 * wj + 8 * nt + g;
        bq[nt][0] = w0 * f64r_at(B, r, 8 * ks + t);
        bq[nt][1] = w1 * f64r_at(B, r, 8 * ks + t + 4);
      }
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        double a[4];
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            a[2 * q + h] = f64r_at(A, 32 * wi + 16 * mt + g + 8 * h, 8 * ks + t + 4 * q);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) dmma_16x8x8(acc[mt][nt], a, bq[nt]);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.empty[st]);
    if (p0 + F64_KC >= prm.P) {
      const int f = (int)(item / prm.ntile);
      double* of = outr + (int64_t)f * prm.npack;
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int i = bi * F64_B + 32 * wi + 16 * mt + g + 8 * (r >> 1);
            const int j = bj * F64_B + 32 * wj + 8 * nt + 2 * t + (r & 1);
            if (i <= j && j < prm.N) of[(int64_t)j * (j + 1) / 2 + i] += acc[mt][nt][r];
          }
    }
  }
  if (failed && warp == 0 && lane == 0) {
    for (int64_t k = c; k < issued; ++k)
      mbar_drain(&sm.full[(int)(k % F64_ST)], (uint32_t)((k / F64_ST) & 1), prm.timeout_ns);
  }
}

// K1r for the `n` frequencies from f0.
static int f64r_launch(const F64Call& q, int f0, int n, int* launches) {
  const int nblk = (q.N + F64_B - 1) / F64_B;
  F64Params prm;
  prm.P = q.P;
  prm.N = q.N;
  prm.W = q.W + (int64_t)f0 * q.ldw;
  prm.ldw = q.ldw;
  prm.nw = n;
  prm.out = nullptr;
  prm.npack = (int64_t)q.N * (q.N + 1) / 2;
  prm.ntile = nblk * (nblk + 1) / 2;
  prm.nitems = (int64_t)prm.ntile * n;
  prm.status = q.status;
  prm.timeout_ns = q.timeout_ns;
  CUtensorMap map;
  const int e = f64_map(&map, q.M, q.ldc, q.P, q.N, F64_B, true);
  if (e) return e;
  const size_t smem = sizeof(F64RSmem) + 1024;
  if (cudaFuncSetAttribute(chi0_fp64_real_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return -2;
  const int grid = (int)std::min<int64_t>(prm.nitems, (int64_t)2 * q.num_sms);
  chi0_fp64_real_kernel<<<grid, F64_THREADS, smem, q.stream>>>(map, prm,
                                                              reinterpret_cast<double*>(q.out) + (int64_t)f0 * prm.npack);
  ++*launches;
  return 0;
}

// Enqueues the FP64 accumulation over one slab of real band-pair products M (ldc, N): ldc
// even, M 16-byte aligned; W as launch_chi0_fp64.
int launch_chi0_fp64_real(spx_ctx* ctx, const double* M, int64_t ldc, int64_t P, int N,
                          const double* W, int64_t ldw, int nw, double* out, cudaStream_t stream,
                          int* launches) {
  if (P <= 0 || N <= 0 || nw <= 0) return SPX_OK;
  const F64Call q{ctx->num_sms, reinterpret_cast<const double2*>(M), ldc, P, N, W, ldw, nw,
                  reinterpret_cast<double2*>(out), (double2*)ctx->part, ctx->part_bytes, ctx->d_status,
                  (uint64_t)(ctx->opt.timeout_ms > 0 ? ctx->opt.timeout_ms : 4000) * 1000000ull, stream};
  const int e = f64_run<F64P_REAL>(q, launches);
  if (e) return set_error(ctx, SPX_ECUDA, "real FP64 accumulation: tensor map or attribute failed (" +
                                              std::to_string(e) + ")");
  return check_cuda(ctx, cudaGetLastError(), "real FP64 accumulation launch");
}

// FP64 tensor-pipe peak: every warp issues back-to-back m16n8k8 DMMAs on register
// operands into eight independent accumulators (no memory traffic in the loop),
// so the rate is the DMMA pipe's own. The sums go to `sink` so nothing is elided.
__global__ void __launch_bounds__(128) dmma_peak_kernel(int iters, double* sink) {
  const int lane = threadIdx.x & 31;
  double a[4], b[2];
#pragma unroll
  for (int k = 0; k < 4; ++k) a[k] = 1.0 + 1e-3 * (lane + k);
  b[0] = 0.5 - 1e-3 * lane;
  b[1] = 0.25 + 1e-3 * lane;
  double d[8][4];
#pragma unroll
  for (int k = 0; k < 8; ++k)
#pragma unroll
    for (int r = 0; r < 4; ++r) d[k][r] = 0.0;
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < 8; ++k) dmma_16x8x8(d[k], a, b);
  }
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k)
#pragma unroll
    for (int r = 0; r < 4; ++r) s += d[k][r];
  sink[blockIdx.x * (int64_t)blockDim.x + threadIdx.x] = s;
}

}  // namespace spx

// Measured FP64 tensor (DMMA) peak of the context's device in TFLOP/s (2 flops
// per MAC), timed with CUDA events on the context stream: one warm-up launch, then
// one launch of 4 CTAs x 4 warps per SM. No counterpart in the reference.
extern "C" int spx_measure_dmma_peak(spx_ctx* ctx, double* tflops) {
  if (!ctx || !tflops) return SPX_EINVAL;
  cudaSetDevice(ctx->device);
  const int blocks = 4 * ctx->num_sms, threads = 128, iters = 20000;
  int rc = spx::ensure_workspace(ctx, sizeof(double) * (size_t)blocks * threads);
  if (rc) return rc;
  double* sink = reinterpret_cast<double*>(ctx->ws);
  cudaEvent_t e0, e1;
  if ((rc = spx::check_cuda(ctx, cudaEventCreate(&e0), "event")) ||
      (rc = spx::check_cuda(ctx, cudaEventCreate(&e1), "event")))
    return rc;
  spx::dmma_peak_kernel<<<blocks, threads, 0, ctx->stream>>>(iters / 10, sink);
  cudaEventRecord(e0, ctx->stream);
  spx::dmma_peak_kernel<<<blocks, threads, 0, ctx->stream>>>(iters, sink);
  cudaEventRecord(e1, ctx->stream);
  rc = spx::check_cuda(ctx, cudaGetLastError(), "dmma_peak_kernel launch");
  if (!rc) rc = spx::check_cuda(ctx, cudaEventSynchronize(e1), "dmma_peak_kernel");
  float ms = 0.f;
  if (!rc) rc = spx::check_cuda(ctx, cudaEventElapsedTime(&ms, e0, e1), "event time");
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  const double macs = 16.0 * 8 * 8 * 8 * (double)iters * (blocks * threads / 32);
  *tflops = 2.0 * macs / (ms * 1e-3) / 1e12;
  return SPX_OK;
}
