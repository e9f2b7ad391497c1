// K2: split-precision band-pair accumulation on the 5th-generation tensor cores.
//
// The sum chi_f(i, j) = sum_p M(p, i) conj(M(p, j)) w(p, f) (src/susceptibility.f:
// 1182-1240 with the HILBERT NONE weights of :950-975) is evaluated as an exact
// integer contraction of 8-bit digit slices (an Ozaki-type error-free split) of
// the weight-folded operand
//
//   A(p, i) = sqrt(|w(p, f)|) M(p, i),   chi_f = A^T diag(sgn w) conj(A),
//
// one operand per frequency for both sides of the product. For every frequency
// whose weights have one sign over the slab (all imaginary-axis HILBERT NONE
// weights) the Gram is A^T conj(A) times that sign, a Hermitian rank-P update
// whose two operands are the same digit planes. Frequencies with weights of both
// signs take B(p, j) = sgn(w(p, f)) A(p, j) as the second operand (its own planes).
// Each value becomes three balanced base-256 digits of one rounded integer,
//
//   A = s sqrt(wmax)/127 * 2^-16 * (d0 2^16 + d1 2^8 + d2),  |d0| <= 127,
//
// with s the largest |Re|, |Im| of the column M(:, i) over the slab of band pairs
// and wmax = max_p |w(p, f)|. The six digit products with t + u <= 2 are summed on
// tcgen05.mma kind::i8 into three int32 accumulators in tensor memory, one per
// order g = t + u, exactly (3 * 128^2 * 32768 < 2^31). Once per slab the epilogue
// forms (D0*256 + D1)*256 + D2 exactly and adds s_i s_j wmax / (127^2 2^16) times
// it (times the sign) to the FP64 output. Weights and scales stay FP64 throughout,
// so near-degenerate pairs keep their FP64 weights.
//
// Error (per element, relative to sqrt(sum_p |w| |M_pi|^2 sum_p |w| |M_pj|^2), which
// is sqrt|chi_ii chi_jj| for one-signed weights): rounding of each operand is half a
// unit of its third digit, 2^-17/127 of its column scale, and the dropped orders
// g >= 3 are of the same size; both enter with the crest factor max|A| sqrt(P)/||A||
// of the folded columns.
//
// A slab runs as statistics (column scales, weights, signs), digit planes, accumulation and,
// when the last items were cut along the pairs over all CTAs, the exact sum of their partial
// tiles; a wide slab's planes are written and accumulated in parts that leave room in L2.
//
// Tile layout: a 64 x 64 complex tile is a 128 x 128 real-stacked product whose rows
// interleave the parts of each mixed-basis function: row 2i holds Re A_i and row
// 2i+1 holds Im A_i (likewise the columns for j). D[2i+c][2j+c'] then holds the four
// real products of (i, j) in two adjacent TMEM lanes, and the epilogue combines
// re = D[2i][2j] + D[2i+1][2j+1], im = D[2i+1][2j] - D[2i][2j+1] by one warp shuffle.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "spx_chain.cuh"
#include "spx_split.cuh"

namespace spx {

constexpr int SP_ST = 4;               // pipeline stages (one CTA per tile)
constexpr int SP_THREADS = 192;        // warp 0 TMA, warp 1 MMA + TMEM, warps 2-5 epilogue
// The one-CTA kernel drains a tile with 8 epilogue warps (warps 2-9; two per TMEM lane
// quarter, each half of the columns): fewer registers per thread, so the operand
// quantizer of the next slab keeps more warps resident beside it on every SM.
constexpr int SP1_EPI = 8;
constexpr int SP_WIDE_BN = 80;  // complex columns of the wide tile (variant 5): N = 160
constexpr int SP1_THREADS = 64 + 32 * SP1_EPI;
constexpr int SP_SMS = 148;   // a B200's SMs, for rules on sizes: scratch does not follow the device's count
constexpr int SP1_REGS = 128;  // 40960 registers: two 96-register quantizer blocks fit beside

// BROWS: real rows of the B tile (the MMA's N): 128 for 64 x 64 complex tiles, 160
// for 64 x 80 (three orders x 160 TMEM columns still fit in 512).
template <int BROWS>
struct __align__(1024) SplitSmemT {
  uint8_t a[SP_ST][SP_SF][SP_PLANE];
  uint8_t b[SP_ST][SP_SF][BROWS * SP_KB];
  uint64_t full[SP_ST];
  uint64_t empty[SP_ST];
  uint64_t tfull, tempty, mdone;
  uint32_t tmem_base;
};
using SplitSmem = SplitSmemT<SP_ROWS>;

struct SplitParams {
  int N;
  int nbr;                // 64-row blocks covering N
  int ntile;
  int nw;
  int nitems;
  int nk;                 // pipeline stages per item (pairs of the slab / 64)
  const double* sA;       // column scales of the slab
  const double* wmax;     // max |w(p, f)| of the slab
  const int* wsgn;        // per frequency: +1 / -1 one-signed weights, 0 both signs
  double* out;            // packed complex output, as doubles
  int64_t npack;
  int whole;              // items dealt whole (all of them without `part`)
  int ncut;               // CTAs that share the stages of the others
  double* part;           // partial tiles [CTA][2 slots][elements], or NULL
  int* status;
  uint64_t timeout_ns;
};

// The items of one CTA of the one-CTA kernels: whole items blockIdx.x, + gridDim.x, ...
// below `whole`, then, in the first `ncut` CTAs, a share of the K stages of the items left over. Those would fill
// a fraction of the SMs for a whole item's time; cut along K they take that fraction of
// it. A partial sum is an exact integer (below 2^49 in magnitude), so adding the parts
// before the scale gives the bits of an uncut item (split_gram_finish_kernel). Measured at
// 403 columns, 12201 pairs, 12 frequencies (336 items on 148 SMs): 375 us uncut with
// 64 x 80 tiles, 270 us cut with 64 x 64 and 9 us for the sum.
struct SplitSeg {
  int item, u, u1, n;
  __device__ __forceinline__ SplitSeg(const SplitParams& p, int cta) {
    item = cta;
    const int64_t tail = (int64_t)(p.nitems - p.whole) * p.nk;   // < 2^31: fewer than 148 items
    u = cta < p.ncut ? (int)(tail * cta / p.ncut) : 0;
    u1 = cta < p.ncut ? (int)(tail * (cta + 1) / p.ncut) : 0;
    n = 0;
  }
  // Next item and its stages [k0, k1); slot -1: the whole item.
  __device__ __forceinline__ bool next(const SplitParams& p, int grid, int* it, int* k0, int* k1, int* slot) {
    if (item < p.whole) {
      *it = item, *k0 = 0, *k1 = p.nk, *slot = -1;
      item += grid;
      return true;
    }
    if (u >= u1) return false;
    const int t = u / p.nk;
    *it = p.whole + t;
    *k0 = u - t * p.nk;
    const int e = min(u1 - t * p.nk, p.nk);
    *k1 = e;
    *slot = (*k0 == 0 && e == p.nk) ? -1 : (n > 0);
    ++n;
    u = t * p.nk + e;
    return true;
  }
};

// Doubles of one partial tile: 64 x BN complex values, or 128 x 2 BN real ones.
__host__ __device__ constexpr int split_part_elems(bool real, int bn) { return (real ? 256 : 128) * bn; }

// This epilogue thread's first value of its CTA's partial tile `slot`; the next ones follow
// 32 SP1_EPI apart.
template <bool REAL, int BN>
__device__ __forceinline__ double* split_part_of(const SplitParams& prm, int slot) {
  return prm.part + ((int64_t)blockIdx.x * 2 + slot) * split_part_elems(REAL, BN) + (threadIdx.x - 64);
}

// Adds a thread's folded values (row bi 64 + 16 q + lane / 2, part lane & 1, NC columns from
// j0 of column block bj) into the packed output. One add per element per launch: launches
// are stream-ordered, so the sum is deterministic, and the reduction needs no read
// round trip.
template <int NC, int BN>
__device__ __forceinline__ void fold_add(int q, int lane, int bi, int bj, int f, const SplitParams& prm,
                                         int j0, const double (&o)[NC]) {
  const int gil = bi * SP_TILE + 16 * q + lane / 2;
  if (gil >= prm.N) return;
  const double fac = fold_row_factor(prm.wsgn[f], prm.sA[gil], prm.wmax[f]);
  double* ob = prm.out + 2 * (int64_t)f * prm.npack + 2 * gil + (lane & 1);
#pragma unroll
  for (int jj = 0; jj < NC; ++jj) {
    const int gj = bj * BN + j0 + jj;
    if (gil <= gj && gj < prm.N) atomicAdd(ob + (int64_t)gj * (gj + 1), fac * prm.sA[gj] * o[jj]);
  }
}

// Adds 16 columns (from j0 of column block bj) of a thread's row of real chi.
template <int BROWS>
__device__ __forceinline__ void real_add16(int q, int lane, int bi, int bj, int f, const SplitParams& prm,
                                           int j0, const double (&T)[16]) {
  const int gi = bi * SP_ROWS + 32 * q + lane;
  if (gi >= prm.N) return;
  const double fac = fold_row_factor(prm.wsgn[f], prm.sA[gi], prm.wmax[f]);
  double* of = prm.out + (int64_t)f * prm.npack + gi;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const int gj = bj * BROWS + j0 + k;
    if (gi <= gj && gj < prm.N) atomicAdd(of + (int64_t)gj * (gj + 1) / 2, fac * prm.sA[gj] * T[k]);
  }
}

// The epilogue of one tile (or of NC of its 64 complex columns, from column j0), run
// by the epilogue warps (warp q reads TMEM lanes 32q..32q+31, i.e. rows
// i = 16q + lane/2, part c = lane & 1). The warp's part of the accumulator is read
// into registers first and released to the MMA warp, so the next item's MMAs overlap
// this tile's reductions into the output.
// A partial item's values go to its slot of `part` instead.
template <int NC = SP_TILE, int BN = SP_TILE, class Release>
__device__ __forceinline__ void fold_epilogue(uint32_t tl, int q, int lane, int bi, int bj, int f,
                                              const SplitParams& prm, Release release, int j0 = 0,
                                              int slot = -1) {
  const int c = lane & 1;
  double o[NC];
#pragma unroll
  for (int cc = 0; cc < NC / 8; ++cc) {
    double T[16];
    load_fold16(tl + (uint32_t)(2 * j0 + 16 * cc), (uint32_t)(2 * BN), T);
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) {
      // both lanes of a row pair send their (., Im_j) product to the other one
      const double pb = __shfl_xor_sync(0xffffffffu, T[2 * jj + 1], 1);
      o[8 * cc + jj] = c == 0 ? T[2 * jj] + pb : T[2 * jj] - pb;
    }
  }
  release();
  if (slot >= 0) {
    double* part = split_part_of<false, BN>(prm, slot);
#pragma unroll
    for (int jj = 0; jj < NC; ++jj) part[jj * (32 * SP1_EPI)] = o[jj];
    return;
  }
  fold_add<NC, BN>(q, lane, bi, bj, f, prm, j0, o);
}

// The -DINV (real) epilogue: columns [j0, j0 + ncol) of a 128 x BROWS tile of real chi,
// TMEM lane = row i of the block, column = j; read and added 16 columns at a time,
// then the accumulator is released.
template <int BROWS, class Release>
__device__ __forceinline__ void real_epilogue(uint32_t tl, int q, int lane, int bi, int bj, int f,
                                              const SplitParams& prm, Release release, int j0,
                                              int ncol, int slot) {
#pragma unroll 1
  for (int cc = 0; cc < ncol / 16; ++cc) {
    double T[16];
    load_fold16(tl + (uint32_t)(j0 + 16 * cc), (uint32_t)BROWS, T);
    if (slot >= 0) {
      double* part = split_part_of<true, BROWS / 2>(prm, slot);
#pragma unroll
      for (int k = 0; k < 16; ++k) part[(16 * cc + k) * (32 * SP1_EPI)] = T[k];
    } else {
      real_add16<BROWS>(q, lane, bi, bj, f, prm, j0 + 16 * cc, T);
    }
  }
  release();
}

// BN: complex columns of a tile (64 or 80; the -DINV form uses 64, i.e. 128 x 128
// real tiles). mapF loads 128-row A boxes, mapB (2 BN)-row B boxes.
template <bool REAL, int BN>
__global__ void __maxnreg__(SP1_REGS)
    split_gram_kernel(const __grid_constant__ CUtensorMap mapF, const __grid_constant__ CUtensorMap mapB,
                      SplitParams prm) {
  constexpr int BROWS = 2 * BN;
  constexpr uint32_t IDESC = sp_idesc(BROWS);
  // the -DINV form: tiles of 128 real rows x BROWS real columns (the same block
  // arithmetic as 64 x BN complex tiles)
  using Smem = SplitSmemT<BROWS>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < SP_ST; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    mbar_init(&sm.tfull, 1);
    mbar_init(&sm.tempty, SP1_EPI);
    mbar_init(&sm.mdone, 1);
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(&sm.tmem_base, SP_TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  release_next();
  await_previous();
  const uint32_t tmem = sm.tmem_base;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 0;
      bool issued[SP_ST];
      uint32_t last_ph[SP_ST];
      for (int s = 0; s < SP_ST; ++s) issued[s] = false, last_ph[s] = 0;
      bool ok = true;
      int item, k0, k1, slot;
      SplitSeg seg(prm, blockIdx.x);
      for (int j = 0; ok && seg.next(prm, gridDim.x, &item, &k0, &k1, &slot); ++j) {
        const int f = item / prm.ntile;
        int bi, bj;
        split_decode_tile_bn<BN>(split_item_tile(item, prm.ntile, gridDim.x), prm.nbr, &bi, &bj);
        const int sg = prm.wsgn[f];
        // a diagonal square tile of a one-signed frequency multiplies A by itself
        const bool same = BN == SP_TILE && sg != 0 && bi == bj;
        const int za = f * SP_SLOT, zb = za + (sg == 0 ? SP_SF : 0);
        for (int ks = k0; ks < k1; ++ks) {
          if (!mbar_wait(&sm.empty[st], ph ^ 1u, prm.timeout_ns, prm.status)) {
            ok = false;
            break;
          }
          // a cut item's stages run forwards in every CTA that has some of them
          const int kc = slot < 0 ? split_k_order(j, ks, prm.nk) : ks;
          mbar_arrive_expect_tx(&sm.full[st], (uint32_t)(SP_SF * (SP_PLANE + (same ? 0 : BROWS * SP_KB))));
          tma_load_4d(&sm.a[st][0][0], &mapF, 0, bi * SP_ROWS, kc, za, &sm.full[st]);
          if (!same) tma_load_4d(&sm.b[st][0][0], &mapB, 0, bj * BROWS, kc, zb, &sm.full[st]);
          issued[st] = true;
          last_ph[st] = ph;
          if (++st == SP_ST) st = 0, ph ^= 1u;
        }
      }
      // copies still landing must finish before this CTA's shared memory goes away
      for (int s = 0; s < SP_ST; ++s)
        if (issued[s]) mbar_drain(&sm.full[s], last_ph[s], prm.timeout_ns);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 0;
      bool committed = false;
      int item, k0, k1, slot;
      SplitSeg seg(prm, blockIdx.x);
      for (int j = 0; seg.next(prm, gridDim.x, &item, &k0, &k1, &slot); ++j) {
        const int f = item / prm.ntile;
        int bi, bj;
        split_decode_tile_bn<BN>(split_item_tile(item, prm.ntile, gridDim.x), prm.nbr, &bi, &bj);
        const bool same = BN == SP_TILE && prm.wsgn[f] != 0 && bi == bj;
        // accumulators free (first item: immediately)
        if (!mbar_wait(&sm.tempty, (uint32_t)(j & 1) ^ 1u, prm.timeout_ns, prm.status)) break;
        tc_fence_after();
        bool ok = true;
        for (int ks = k0; ks < k1; ++ks) {
          if (!mbar_wait(&sm.full[st], ph, prm.timeout_ns, prm.status)) {
            ok = false;
            break;
          }
          tc_fence_after();
          // order g = t + u lives at TMEM columns [BROWS g, BROWS g + BROWS); the
          // first product of every order in an item (first K step) overwrites it
#pragma unroll
          for (int kk = 0; kk < SP_NKS; ++kk) {
            uint64_t da[SP_SF], db[SP_SF];
#pragma unroll
            for (int t = 0; t < SP_SF; ++t) {
              da[t] = desc_sw64(&sm.a[st][t][0]) + (uint64_t)(kk * 2);
              db[t] = same ? da[t] : desc_sw64(&sm.b[st][t][0]) + (uint64_t)(kk * 2);
            }
            const uint32_t kacc = (ks > k0 || kk > 0);
            mma_i8<1>(tmem + 0 * BROWS, da[0], db[0], IDESC, kacc);
            mma_i8<2>(tmem + 1 * BROWS, da[0], db[1], IDESC, kacc);
            mma_i8<3>(tmem + 2 * BROWS, da[0], db[2], IDESC, kacc);
            mma_i8<1>(tmem + 1 * BROWS, da[1], db[0], IDESC, 1u);
            mma_i8<3>(tmem + 2 * BROWS, da[1], db[1], IDESC, 1u);
            mma_i8<0>(tmem + 2 * BROWS, da[2], db[0], IDESC, 1u);
          }
          tc_commit(&sm.empty[st]);  // stage free once these MMAs have read it
          committed = true;
          if (++st == SP_ST) st = 0, ph ^= 1u;
        }
        if (!ok) break;
        tc_commit(&sm.tfull);  // accumulators complete
      }
      // every MMA issued by this thread must retire before TMEM is released: a
      // commit issued now arrives once all of them are done
      if (committed) {
        tc_commit(&sm.mdone);
        mbar_drain(&sm.mdone, 0u, prm.timeout_ns);
      }
    }
  } else {
    // ---- epilogue: SP1_EPI warps, SP1_EPI / 4 per TMEM lane quarter (column ranges) ----
    const int q = warp & 3, h = (warp - 2) >> 2;
    const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
    int item, k0, k1, slot;
    SplitSeg seg(prm, blockIdx.x);
    for (int j = 0; seg.next(prm, gridDim.x, &item, &k0, &k1, &slot); ++j) {
      if (!mbar_wait_idle(&sm.tfull, (uint32_t)(j & 1), prm.timeout_ns, prm.status)) break;
      tc_fence_after();
      const int f = item / prm.ntile;
      int bi, bj;
      split_decode_tile_bn<BN>(split_item_tile(item, prm.ntile, gridDim.x), prm.nbr, &bi, &bj);
      auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.tempty);
      };
      constexpr int NC = BN * 4 / SP1_EPI;  // complex columns per epilogue warp
      if constexpr (REAL) real_epilogue<BROWS>(tl, q, lane, bi, bj, f, prm, release, 2 * NC * h, 2 * NC, slot);
      else fold_epilogue<NC, BN>(tl, q, lane, bi, bj, f, prm, release, NC * h, slot);
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, SP_TMEM_COLS);
}

// One CTA per boundary between the stage ranges of CTAs c - 1 and c (grid.x = CTAs of the
// accumulation - 1) and 16 or 8 columns of a thread's share (grid.y): the first boundary
// inside an item adds the item's partial tiles (exact) in CTA order, then the scaled
// sum into the output as the uncut epilogue does.
template <bool REAL>
constexpr int split_finish_step() { return REAL ? 16 : 8; }
template <bool REAL, int BN>
__global__ void __launch_bounds__(32 * SP1_EPI) split_gram_finish_kernel(SplitParams prm, int grid) {
  await_previous();
  const int64_t tail = (int64_t)(prm.nitems - prm.whole) * prm.nk;
  const int c = blockIdx.x + 1;
  const int64_t u = tail * c / prm.ncut;
  const int64_t t0 = u / prm.nk * prm.nk, t1 = t0 + prm.nk;
  if (u == t0 || u >= tail || tail * (c - 1) / prm.ncut > t0) return;
  const int item = prm.whole + (int)(t0 / prm.nk);
  const int f = item / prm.ntile;
  int bi, bj;
  split_decode_tile_bn<BN>(split_item_tile(item, prm.ntile, grid), prm.nbr, &bi, &bj);
  const int warp = (threadIdx.x >> 5) + 2, lane = threadIdx.x & 31;   // the epilogue's warp numbers
  const int q = warp & 3, h = (warp - 2) >> 2;
  constexpr int NC = BN * 4 / SP1_EPI, STEP = split_finish_step<REAL>();
  const int v0 = blockIdx.y * STEP;
  double o[STEP];
#pragma unroll
  for (int v = 0; v < STEP; ++v) o[v] = 0.0;
  for (int k = c - 1; k < prm.ncut; ++k) {
    const int64_t s = tail * k / prm.ncut;
    if (s >= t1) break;
    if (tail * (k + 1) / prm.ncut == s) continue;   // an empty range
    // the item is a CTA's first segment when its range starts inside it
    const double* pp = prm.part + ((int64_t)k * 2 + (s >= t0 ? 0 : 1)) * split_part_elems(REAL, BN) +
                       (int64_t)v0 * (32 * SP1_EPI) + threadIdx.x;
#pragma unroll
    for (int v = 0; v < STEP; ++v) o[v] += pp[v * (32 * SP1_EPI)];
  }
  if constexpr (REAL) real_add16<2 * BN>(q, lane, bi, bj, f, prm, 2 * NC * h + v0, o);
  else fold_add<STEP, BN>(q, lane, bi, bj, f, prm, NC * h + v0, o);
}

// CTAs that share the stages of the items left over by whole rounds of `num_sms` CTAs; 0 when
// these stay whole. A share is about the root of an item's `nk` stages at least: a stage takes
// 0.55-0.6 us, and an item's partial tiles are added one after the other at about the same time
// each. Cutting pays when it saves this many of the last round's stages: it costs the partial
// tiles' way through memory and one short launch, 20 us with complex tiles (403 columns, 12
// frequencies: 40 of 336 items left), 40 us with the twice as large real ones.
int split_cut_ctas(int nitems, int nk, int num_sms, bool real) {
  const int64_t left = nitems % num_sms, tail = left * nk;
  if (left == 0) return 0;
  int64_t share = 8;
  while (share * share < nk) ++share;
  const int64_t even = (tail + num_sms - 1) / num_sms;
  if (nk - std::max(share, even) < (real ? 128 : 64)) return 0;
  return (int)std::min<int64_t>(num_sms, tail / share);
}

// ---------------------------------------------------------------------------
// CTA-pair form: one tcgen05.mma.cta_group::2 (M = 256) covers two 64 x 64 complex
// tiles stacked in i. Each CTA of the cluster stages its own A tile (128 rows) and
// half of the shared B tile (64 rows: CTA 0 the columns j of the first 32, CTA 1
// the next 32); the leader CTA issues the MMAs, which read both CTAs' shared memory
// and write each CTA's own TMEM. Every completion that crosses the pair is an
// explicit remote arrive or commit (no multicast).

constexpr int SP2_ST = 5;
constexpr int SP2_BROWS = SP_ROWS / 2;          // B rows staged per CTA
constexpr int SP2_BPLANE = SP2_BROWS * SP_KB;   // 4096 bytes
constexpr uint32_t SP2_IDESC = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(SP_ROWS / 8) << 17) |
                               ((uint32_t)(2 * SP_ROWS / 16) << 24);   // M = 256, N = 128

struct __align__(1024) Split2Smem {
  uint8_t a[SP2_ST][SP_SF][SP_PLANE];
  uint8_t b[SP2_ST][SP_SF][SP2_BPLANE];
  uint64_t full[SP2_ST];   // leader: both CTAs' bytes of a stage have landed
  uint64_t empty[SP2_ST];  // each CTA: the MMAs have read the stage
  uint64_t tfull;          // each CTA: accumulators ready
  uint64_t tempty;         // leader: both CTAs' epilogues have drained TMEM (8 warps)
  uint64_t mdone;
  uint32_t tmem_base;
};

// Pair tile t -> (bI, bJ): i-blocks of 128 (two 64-blocks), j-blocks of 64, with
// 2 bI <= bJ; column-major over bJ.
__device__ __forceinline__ void pair_decode_tile(int t, int* bI, int* bJ) {
  int j = 0, c = 0;
  while (c + j / 2 + 1 <= t) {
    c += j / 2 + 1;
    ++j;
  }
  *bJ = j;
  *bI = t - c;
}

__global__ void __launch_bounds__(SP_THREADS, 1)
    split_gram2_kernel(const __grid_constant__ CUtensorMap mapF,
                       const __grid_constant__ CUtensorMap mapFh, SplitParams prm) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  Split2Smem& sm = *reinterpret_cast<Split2Smem*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int cid = (int)cluster_id_x(), ncl = (int)nclusters_x();

  if (threadIdx.x == 0) {
    for (int s = 0; s < SP2_ST; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    mbar_init(&sm.tfull, 1);
    mbar_init(&sm.tempty, 8);
    mbar_init(&sm.mdone, 1);
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc2(&sm.tmem_base, SP_TMEM_COLS);
  tc_fence_before();
  cluster_sync();  // both CTAs' barriers initialised and TMEM allocated
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 0;
      bool issued[SP2_ST];
      uint32_t last_ph[SP2_ST];
      for (int q = 0; q < SP2_ST; ++q) issued[q] = false, last_ph[q] = 0;
      // Cursor over this cluster's (item, stage) sequence; it advances by increments
      // and decodes a tile only when it enters a new item.
      struct Cursor {
        int item, ks, ya, yb, za, zb, j;
      };
      auto enter = [&](Cursor& u) {
        int bI, bJ;
        pair_decode_tile(u.item % prm.ntile, &bI, &bJ);
        const int f = u.item / prm.ntile;
        u.ya = (2 * bI + (int)rank) * SP_ROWS;
        u.yb = bJ * SP_ROWS + (int)rank * SP2_BROWS;
        u.za = f * SP_SLOT;
        u.zb = u.za + (prm.wsgn[f] == 0 ? SP_SF : 0);
      };
      auto advance = [&](Cursor& u) {
        if (++u.ks == prm.nk) {
          u.ks = 0;
          u.item += ncl;
          ++u.j;
          if (u.item < prm.nitems) enter(u);
        }
      };
      Cursor ld{cid, 0, 0, 0, 0, 0, 0};
      if (cid < prm.nitems) enter(ld);
      while (ld.item < prm.nitems) {
        if (!mbar_wait(&sm.empty[st], ph ^ 1u, prm.timeout_ns, prm.status)) break;
        const uint32_t lead_full = mapa_shared(smem_u32(&sm.full[st]), 0);
        if (rank == 0)
          mbar_arrive_expect_tx(&sm.full[st], (uint32_t)(2 * SP_SF * (SP_PLANE + SP2_BPLANE)));
        const int kc = split_k_order(ld.j, ld.ks, prm.nk);
        tma_load_4d_pair(&sm.a[st][0][0], &mapF, 0, ld.ya, kc, ld.za, lead_full);
        tma_load_4d_pair(&sm.b[st][0][0], &mapFh, 0, ld.yb, kc, ld.zb, lead_full);
        advance(ld);
        issued[st] = true;
        last_ph[st] = ph;
        if (++st == SP2_ST) st = 0, ph ^= 1u;
      }
      if (rank == 0) {
        // the leader's stage barriers count both CTAs' bytes
        for (int q = 0; q < SP2_ST; ++q)
          if (issued[q]) mbar_drain(&sm.full[q], last_ph[q], prm.timeout_ns);
      } else {
        // the peer cannot poll the leader's barrier: give its last copies a bounded
        // grace period to land (they complete in microseconds)
        const uint64_t t0 = global_ns();
        while (global_ns() - t0 < 200000ull) {
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (rank == 0 && lane == 0) {
      int st = 0;
      uint32_t ph = 0;
      int j = 0;
      bool committed = false;
      const uint32_t peer_tfull = mapa_shared(smem_u32(&sm.tfull), 1);
      for (int item = cid; item < prm.nitems; item += ncl, ++j) {
        if (!mbar_wait(&sm.tempty, (uint32_t)(j & 1) ^ 1u, prm.timeout_ns, prm.status)) break;
        tc_fence_after();
        bool ok = true;
        for (int ks = 0; ks < prm.nk; ++ks) {
          if (!mbar_wait(&sm.full[st], ph, prm.timeout_ns, prm.status)) {
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < SP_NKS; ++kk) {
            uint64_t da[SP_SF], db[SP_SF];
#pragma unroll
            for (int t = 0; t < SP_SF; ++t) {
              da[t] = desc_sw64(&sm.a[st][t][0]) + (uint64_t)(kk * 2);
              db[t] = desc_sw64(&sm.b[st][t][0]) + (uint64_t)(kk * 2);
            }
            const uint32_t k0 = (ks > 0 || kk > 0);
            mma2_i8<1>(tmem + 0 * 128, da[0], db[0], SP2_IDESC, k0);
            mma2_i8<2>(tmem + 1 * 128, da[0], db[1], SP2_IDESC, k0);
            mma2_i8<3>(tmem + 2 * 128, da[0], db[2], SP2_IDESC, k0);
            mma2_i8<1>(tmem + 1 * 128, da[1], db[0], SP2_IDESC, 1u);
            mma2_i8<3>(tmem + 2 * 128, da[1], db[1], SP2_IDESC, 1u);
            mma2_i8<0>(tmem + 2 * 128, da[2], db[0], SP2_IDESC, 1u);
          }
          // the stage is free in both CTAs once these MMAs have read it
          tc_commit2(smem_u32(&sm.empty[st]));
          tc_commit2(mapa_shared(smem_u32(&sm.empty[st]), 1));
          committed = true;
          if (++st == SP2_ST) st = 0, ph ^= 1u;
        }
        if (!ok) break;
        tc_commit2(smem_u32(&sm.tfull));
        tc_commit2(peer_tfull);
      }
      if (committed) {
        tc_commit2(smem_u32(&sm.mdone));
        mbar_drain(&sm.mdone, 0u, prm.timeout_ns);
      }
    }
  } else {
    // ---------------- epilogue (both CTAs): this CTA's 64 x 64 tile ----------------
    const int q = warp & 3;
    const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16);
    const uint32_t lead_tempty = mapa_shared(smem_u32(&sm.tempty), 0);
    int j = 0;
    for (int item = cid; item < prm.nitems; item += ncl, ++j) {
      if (!mbar_wait_idle(&sm.tfull, (uint32_t)(j & 1), prm.timeout_ns, prm.status)) break;
      tc_fence_after();
      const int f = item / prm.ntile;
      int bI, bJ;
      pair_decode_tile(item % prm.ntile, &bI, &bJ);
      const int bi = 2 * bI + (int)rank;
      auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (rank == 0) mbar_arrive(&sm.tempty);
          else mbar_arrive_cluster(lead_tempty);
        }
      };
      // a tile wholly below the diagonal or past N has nothing to store
      if (bi <= bJ && bi * SP_TILE < prm.N) fold_epilogue(tl, q, lane, bi, bJ, f, prm, release);
      else release();
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();  // neither CTA leaves while the pair's MMAs may read its shared memory
  tc_fence_after();
  if (warp == 1) tmem_dealloc2(tmem, SP_TMEM_COLS);
}

// ---------------------------------------------------------------------------
// operand preparation

// Maximum over the CTA of a non-negative value, for every thread.
__device__ __forceinline__ double block_max(double m, double* red) {
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  m = red[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, red[w]);
  return m;
}

// Statistics of one slab, one launch of clusters of SPS_CL CTAs:
//   * the first `ncol` CTAs (N rounded up to whole clusters): the column scales
//     sA[i] = max_p max(|Re M(p,i)|, |Im M(p,i)|), one column each;
//   * then one cluster per frequency f: wmax[f] = max_p |w(p, f)|, the sign code wsgn[f]
//     (+1 all weights >= 0, -1 all <= 0, 0 both signs), and the folded factors
//     G[f][p] = sgn(w) sqrt(|w| / wmax) * 127 * 2^16 (0 past the slab's end), each CTA an
//     eighth of the slab, the maximum and signs shared through the cluster's shared memory.
// The factors cost a division and a square root each, and a frequency's were one CTA's
// work: 102 us for 32768 pairs x 24 frequencies, on the critical path before the first
// accumulation. With ediff the weights are formed here (HILBERT NONE), else read from W.
// Measured at 403 columns, 12201 pairs, 12 frequencies: 18 us, against 70 us in three
// launches (weights, column scales, frequency statistics).
constexpr int SPS_CL = 8, SPS_THREADS = 256;
struct SplitStat {
  const double* W;       // caller's weights (ldw, nw), or NULL:
  int64_t ldw;
  const double* ediff;   // HILBERT NONE weights of these energy differences
  const double* wscale;
  double scale_all;
  const double* omega;
};
template <bool REAL>
__global__ void __launch_bounds__(SPS_THREADS) __cluster_dims__(SPS_CL, 1, 1)
    split_stat_kernel(const double* __restrict__ M, int64_t ldc, int64_t p0, int len, int lenp, int N,
                      int ncol, SplitStat src, double* __restrict__ sA, double* __restrict__ wmax,
                      int* __restrict__ wsgn, double* __restrict__ G) {
  __shared__ double red[SPS_THREADS / 32];
  __shared__ double share_m;
  __shared__ int share_s;
  release_next();
  if ((int)blockIdx.x < ncol) {
    const int i = blockIdx.x;
    if (i >= N) return;   // whole clusters take this branch, and none of it synchronises them
    double m = 0.0;
    if constexpr (REAL) {
      const double* col = M + (int64_t)i * ldc + p0;
#pragma unroll 4
      for (int p = threadIdx.x; p < len; p += SPS_THREADS) m = fmax(m, fabs(__ldg(col + p)));
    } else {
      const double2* col = reinterpret_cast<const double2*>(M) + (int64_t)i * ldc + p0;
#pragma unroll 4
      for (int p = threadIdx.x; p < len; p += SPS_THREADS) {
        const double2 v = __ldg(col + p);
        m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
      }
    }
    m = block_max(m, red);
    if (threadIdx.x == 0) sA[i] = m;
    return;
  }
  const int f = ((int)blockIdx.x - ncol) / SPS_CL, r = ((int)blockIdx.x - ncol) % SPS_CL;
  const double om = src.W ? 0.0 : src.omega[f];
  auto weight = [&](int p) {
    if (src.W) return src.W[(int64_t)f * src.ldw + p0 + p];
    return hilbert_none_weight(src.ediff[p0 + p], om, (src.wscale ? src.wscale[p0 + p] : 1.0) * src.scale_all);
  };
  // the CTA's pairs, in whole 64-pair blocks of the slab
  const int nb = lenp / SP_KB, a = (int)((int64_t)nb * r / SPS_CL) * SP_KB,
            e = (int)((int64_t)nb * (r + 1) / SPS_CL) * SP_KB;
  double m = 0.0;
  int sg = 0;   // bit 0: a positive weight, bit 1: a negative one
  for (int p = a + threadIdx.x; p < min(e, len); p += SPS_THREADS) {
    const double w = weight(p);
    m = fmax(m, fabs(w));
    sg |= (w > 0.0 ? 1 : 0) | (w < 0.0 ? 2 : 0);
  }
  m = block_max(m, red);
  sg = __syncthreads_or(sg & 1) | (__syncthreads_or(sg & 2) ? 2 : 0);
  if (threadIdx.x == 0) share_m = m, share_s = sg;
  cluster_sync();
  double wm = 0.0;
  sg = 0;
#pragma unroll
  for (int k = 0; k < SPS_CL; ++k) {
    wm = fmax(wm, ld_cluster_f64(&share_m, k));
    sg |= ld_cluster_s32(&share_s, k);
  }
  if (r == 0 && threadIdx.x == 0) {
    wmax[f] = wm;
    wsgn[f] = sg == 3 ? 0 : (sg == 2 ? -1 : 1);
  }
  double* gf = G + (int64_t)f * lenp;
  for (int p = a + threadIdx.x; p < e; p += SPS_THREADS) gf[p] = p < len ? fold_factor(weight(p), wm) : 0.0;
  cluster_sync();   // no CTA leaves while another may still read its maximum
}

// One thread = one complex column i and 8 consecutive pairs of the slab. Digit
// planes are stored [plane][k-block of 64 pairs][row][64 bytes]; a warp holds 4
// consecutive columns x the eight 8-pair pieces of one k-block, so its stores cover
// 8 adjacent rows x 64 bytes, and the TMA box (64 B, rows, 1 k-block, planes) lands
// as [plane][row][64 B] in shared memory. Rows interleave the parts: column i ->
// rows 128 (i / 64) + 2 (i % 64) (Re) and the next one (Im). For frequency f the
// planes f*6 + t hold the digits t of round(x |G| / s) (the folded operand), and,
// when the frequency's weights have both signs, planes f*6 + 3 + t those of
// round(x G / s). A block is 16 columns x one 64-pair k-block; the block stages the
// folded factors of its 64 pairs (SPQ_FCH frequencies at a time) in shared memory,
// so the frequency loop waits on no L2 round trip. 24 frequencies are 12 KB, which does not
// fit on an SM beside an accumulation CTA (217 KB with 64 x 80 tiles): the next part's
// planes are written where the accumulation's last round leaves SMs idle, and after it.
// Side by side on every SM (8 frequencies at a time) both got slower: real form, 900
// columns, 8192 pairs, 712 us for both against 420 + 139 us one after the other. The kernel is bound by the HBM
// writes of the planes; 96 registers keep five blocks per SM. sA, wsgn and G are still being
// written when the first blocks start (spx_chain.cuh): ordinary loads after the wait.
constexpr int SPQ_FCH = 24;
__global__ void __maxnreg__(96)
    split_quantize_kernel(const double2* __restrict__ M, int64_t ldc, int64_t p0, int len,
                          int nchunk, int N, int npad, int64_t R, int64_t Ps, int nw,
                          const double* sA, const int* wsgn, const double* G, int ldg, int8_t* __restrict__ F) {
  __shared__ __align__(16) double gs[SPQ_FCH][SP_KB];
  __shared__ int ss[SPQ_FCH];
  // thread -> (k-block, column group of 4, eighth of the k-block, column in group); the
  // 4 warps of a block share the k-block (npad / 4 is a multiple of 4)
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool active = tid < (int64_t)npad * nchunk * 2;
  const int ngroup = npad / 4;
  const int lane4 = (int)(tid & 3), eighth = (int)((tid >> 2) & 7);
  const int64_t rest = tid >> 5;
  const int i = (int)(rest % ngroup) * 4 + lane4;
  const int64_t kb = ((blockIdx.x * (int64_t)blockDim.x) >> 5) / ngroup;  // the block's k-block
  const int p = (int)(kb * SP_KB) + eighth * 8;
  const int64_t nkb = Ps / SP_KB;
  // planes are nkb * R * 64 bytes apart
  const int64_t pstride = nkb * R * SP_KB;
  const int64_t o_re = (kb * R + split_row_re(i)) * SP_KB + eighth * 8;
  const bool col_ok = active && i < N;
  const double2* col = M + (int64_t)(col_ok ? i : 0) * ldc + p0;
  double xr[8], xi[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    double2 v = make_double2(0.0, 0.0);
    if (col_ok && p + k < len) v = __ldg(col + p + k);
    xr[k] = v.x;
    xi[k] = v.y;
  }
  release_next();
  await_previous();
  const double s = col_ok ? sA[i] : 0.0;
  const double inv = s > 0.0 ? 1.0 / s : 0.0;
  for (int f0 = 0; f0 < nw; f0 += SPQ_FCH) {
    const int nf = min(SPQ_FCH, nw - f0);
    __syncthreads();  // the previous chunk's factors are consumed
    // 16-byte chunk c = 4 e + j (eighth e, chunk j of its 8 pairs) is kept at
    // 4 e + (j ^ ((e >> 1) & 3)): the eight eighths a warp reads at once fall in
    // distinct banks
    for (int e = threadIdx.x; e < nf * (SP_KB / 2); e += blockDim.x) {
      const int f = e / (SP_KB / 2), c = e - f * (SP_KB / 2);
      const int ce = c >> 2, cj = c & 3;
      reinterpret_cast<double2*>(&gs[f][0])[4 * ce + (cj ^ ((ce >> 1) & 3))] =
          reinterpret_cast<const double2*>(G + (int64_t)(f0 + f) * ldg + kb * SP_KB)[c];
    }
    for (int f = threadIdx.x; f < nf; f += blockDim.x) ss[f] = wsgn[f0 + f];
    __syncthreads();
    if (!active) continue;
#pragma unroll 1
    for (int f = 0; f < nf; ++f) {
      const bool mixed = ss[f] == 0;
      const double2* gq2 = reinterpret_cast<const double2*>(&gs[f][eighth * 8]);
      const int sw = (eighth >> 1) & 3;
      uint32_t ar[SP_SF][2], ai[SP_SF][2], br[SP_SF][2], bim[SP_SF][2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t yr[4], yi[4], pr[SP_SF], pi[SP_SF];
        double gq[4];
        const double2 g01 = gq2[(2 * q) ^ sw], g23 = gq2[(2 * q + 1) ^ sw];
        gq[0] = g01.x * inv, gq[1] = g01.y * inv, gq[2] = g23.x * inv, gq[3] = g23.y * inv;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const double ga = fabs(gq[e]);
          yr[e] = round_mul(xr[4 * q + e], ga);
          yi[e] = round_mul(xi[4 * q + e], ga);
        }
        digit_planes<SP_SF>(yr, pr);
        digit_planes<SP_SF>(yi, pi);
#pragma unroll
        for (int t = 0; t < SP_SF; ++t) ar[t][q] = pr[t], ai[t][q] = pi[t];
        if (mixed) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (gq[e] < 0.0) yr[e] = 0u - yr[e], yi[e] = 0u - yi[e];
          digit_planes<SP_SF>(yr, pr);
          digit_planes<SP_SF>(yi, pi);
#pragma unroll
          for (int t = 0; t < SP_SF; ++t) br[t][q] = pr[t], bim[t][q] = pi[t];
        }
      }
#pragma unroll
      for (int t = 0; t < SP_SF; ++t) {
        const int64_t plane = (int64_t)(f0 + f) * SP_SLOT + t;
        *reinterpret_cast<uint2*>(F + o_re + plane * pstride) = make_uint2(ar[t][0], ar[t][1]);
        *reinterpret_cast<uint2*>(F + o_re + SP_KB + plane * pstride) = make_uint2(ai[t][0], ai[t][1]);
      }
      if (mixed) {
#pragma unroll
        for (int t = 0; t < SP_SF; ++t) {
          const int64_t plane = (int64_t)(f0 + f) * SP_SLOT + SP_SF + t;
          *reinterpret_cast<uint2*>(F + o_re + plane * pstride) = make_uint2(br[t][0], br[t][1]);
          *reinterpret_cast<uint2*>(F + o_re + SP_KB + plane * pstride) = make_uint2(bim[t][0], bim[t][1]);
        }
      }
    }
  }
}

// -DINV (real M): digit planes with one plane row per column (rows 128 b .. 128 b + 127
// hold the columns of 128-block b). A thread is one column and 16 pairs, a warp 8 columns
// x the four quarters of a 64-pair block, a block 32 columns; the factors of the block's
// 64 pairs are staged in shared memory as in the complex form (16-byte chunk c = 8 q + j
// of quarter q at 8 q + (j ^ 2 q): the quarters a warp reads at once fall in distinct
// banks). Bound by the planes' writes: 900 columns, 32768 pairs, 24 frequencies 826 ->
// 525 us (4.8 TB/s).
__global__ void __launch_bounds__(128, 5)
    split_quantize_real_kernel(const double* __restrict__ M, int64_t ldc, int64_t p0, int len,
                               int nchunk, int N, int npad, int64_t R, int64_t Ps, int nw,
                               const double* sA, const int* wsgn, const double* G, int ldg, int8_t* __restrict__ F) {
  __shared__ __align__(16) double gs[SPQ_FCH][SP_KB];
  __shared__ int ss[SPQ_FCH];
  const int ngroup = npad / 8;   // a multiple of 16, so a block's 4 warps share the k-block
  const int64_t warp0 = blockIdx.x * 4ll;
  const int64_t kb = warp0 / ngroup;
  const int lane8 = threadIdx.x & 7, quarter = (threadIdx.x >> 3) & 3;
  const int i = (int)((warp0 + (threadIdx.x >> 5)) % ngroup) * 8 + lane8;
  const int p = (int)(kb * SP_KB) + quarter * 16;
  const int64_t pstride = (Ps / SP_KB) * R * SP_KB, o = (kb * R + i) * SP_KB + quarter * 16;
  const bool col_ok = i < N;
  const double* col = M + (int64_t)(col_ok ? i : 0) * ldc + p0;
  double x[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) x[k] = (col_ok && p + k < len) ? __ldg(col + p + k) : 0.0;
  release_next();
  await_previous();
  const double s = col_ok ? sA[i] : 0.0;
  const double inv = s > 0.0 ? 1.0 / s : 0.0;
  for (int f0 = 0; f0 < nw; f0 += SPQ_FCH) {
    const int nf = min(SPQ_FCH, nw - f0);
    __syncthreads();   // the previous chunk's factors are consumed
    for (int e = threadIdx.x; e < nf * (SP_KB / 2); e += blockDim.x) {
      const int f = e / (SP_KB / 2), c = e - f * (SP_KB / 2), q = c >> 3, j = c & 7;
      reinterpret_cast<double2*>(&gs[f][0])[8 * q + (j ^ (2 * q))] =
          reinterpret_cast<const double2*>(G + (int64_t)(f0 + f) * ldg + kb * SP_KB)[c];
    }
    for (int f = threadIdx.x; f < nf; f += blockDim.x) ss[f] = wsgn[f0 + f];
    __syncthreads();
#pragma unroll 1
    for (int f = 0; f < nf; ++f) {
      const bool mixed = ss[f] == 0;
      const double2* gq = reinterpret_cast<const double2*>(&gs[f][0]) + 8 * quarter;
      uint32_t a[SP_SF][4], b[SP_SF][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double2 g01 = gq[(2 * q) ^ (2 * quarter)], g23 = gq[(2 * q + 1) ^ (2 * quarter)];
        const double g[4] = {g01.x * inv, g01.y * inv, g23.x * inv, g23.y * inv};
        uint32_t y[4], pd[SP_SF];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] = round_mul(x[4 * q + e], fabs(g[e]));
        digit_planes<SP_SF>(y, pd);
#pragma unroll
        for (int t = 0; t < SP_SF; ++t) a[t][q] = pd[t];
        if (mixed) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (g[e] < 0.0) y[e] = 0u - y[e];
          digit_planes<SP_SF>(y, pd);
#pragma unroll
          for (int t = 0; t < SP_SF; ++t) b[t][q] = pd[t];
        }
      }
#pragma unroll
      for (int t = 0; t < SP_SF; ++t)
        *reinterpret_cast<uint4*>(F + o + ((int64_t)(f0 + f) * SP_SLOT + t) * pstride) =
            make_uint4(a[t][0], a[t][1], a[t][2], a[t][3]);
      if (mixed) {
#pragma unroll
        for (int t = 0; t < SP_SF; ++t)
          *reinterpret_cast<uint4*>(F + o + ((int64_t)(f0 + f) * SP_SLOT + SP_SF + t) * pstride) =
              make_uint4(b[t][0], b[t][1], b[t][2], b[t][3]);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// Generic tiled tensor map (no context): 0 on success, -1 without the driver entry
// point, else the driver's error code.
int encode_tmap(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* base,
                const uint64_t* dims, const uint64_t* strides, const uint32_t* box,
                CUtensorMapSwizzle swz) {
  auto enc = get_encode();
  if (!enc) return -1;
  cuuint64_t d[5], st[4];
  cuuint32_t b[5], es[5];
  for (int i = 0; i < rank; ++i) {
    d[i] = dims[i];
    b[i] = box[i];
    es[i] = 1;
    if (i + 1 < rank) st[i] = strides[i];
  }
  return (int)enc(map, type, (cuuint32_t)rank, const_cast<void*>(base), d, st, b, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

int make_tmap_u8_3d(spx_ctx* ctx, CUtensorMap* map, const void* base, uint64_t d0, uint64_t d1,
                    uint64_t d2, uint64_t s1, uint64_t s2, uint32_t b0, uint32_t b1, uint32_t b2,
                    CUtensorMapSwizzle swz) {
  auto enc = get_encode();
  if (!enc) return set_error(ctx, SPX_ECUDA, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[3] = {d0, d1, d2};
  cuuint64_t strides[2] = {s1, s2};
  cuuint32_t box[3] = {b0, b1, b2};
  cuuint32_t es[3] = {1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides,
                   box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return set_error(ctx, SPX_ECUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return SPX_OK;
}

int make_tmap_u8_4d(spx_ctx* ctx, CUtensorMap* map, const void* base, const uint64_t dims[4],
                    const uint64_t strides[3], const uint32_t box[4], CUtensorMapSwizzle swz) {
  auto enc = get_encode();
  if (!enc) return set_error(ctx, SPX_ECUDA, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t d[4] = {dims[0], dims[1], dims[2], dims[3]};
  cuuint64_t st[3] = {strides[0], strides[1], strides[2]};
  cuuint32_t b[4] = {box[0], box[1], box[2], box[3]};
  cuuint32_t es[4] = {1, 1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(base), d, st, b, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return set_error(ctx, SPX_ECUDA, "cuTensorMapEncodeTiled (4-D) failed: " + std::to_string((int)r));
  return SPX_OK;
}

struct SplitLayout {
  int64_t Ps, most, R;   // pairs of a slab, the most pairs of a part, plane rows
  int64_t pairs;         // pairs of planes reserved, for all operand buffers together
  int nblk, nstat;       // sets of slab statistics
  size_t f_bytes, g_bytes, s_bytes, w_bytes, sg_bytes;
  size_t bytes() const { return f_bytes + nstat * (g_bytes + s_bytes + w_bytes + sg_bytes) + 1024; }
  // Pairs of a part of a slab of `len` pairs.
  int64_t part(int64_t len) const {
    const int64_t n = std::max<int64_t>((len + most - 1) / most, 1);
    return (int64_t)align_up((size_t)((len + n - 1) / n), SP_KB);
  }
};

// Tiles of one frequency on 64 x BN complex tiles (the -DINV form: 128 x 2 BN real ones,
// nbr its 128-row blocks and n the columns in halves).
static int split_ntile(int n, int bn, int nbr) {
  int t = 0;
  for (int bj = 0; bj * bn < n; ++bj) t += split_rows_of(bj, bn, nbr);
  return t;
}

// One-CTA tile shape of an untuned call: the shape whose tiles take less tensor-pipe time. An MMA
// of N = 160 takes 1.10 times the time of one of N = 128 (which is bound by the instruction
// rate), so 64 x 80 tiles win (1.13 fewer of them at 1200 columns: 739 against 705 TFLOP/s)
// unless their last column block is nearly empty (403 columns: 28 tiles of either shape).
// Tiles count in rounds of the SMs, a cut last round (`cut`: partial tiles can be had) as its
// fraction and the 36 or 72 stages that its sum takes: 320 columns, 10 frequencies are 140
// wide tiles or 150 square ones, 110 and 114 us at 4160 pairs (65 stages), where a cut does not pay.
static bool split_wide(int n, int nbr, int nw, int64_t nk, int num_sms, bool real, bool cut) {
  auto rounds = [&](int bn) {
    const int items = split_ntile(n, bn, nbr) * nw;
    if (cut && split_cut_ctas(items, (int)nk, num_sms, real))
      return (double)items / num_sms + (real ? 72.0 : 36.0) / (double)nk;
    return (double)((items + num_sms - 1) / num_sms);
  };
  return 1.10 * rounds(SP_WIDE_BN) < rounds(SP_TILE);
}

// Most pairs of a part: a slab's scales and factors hold for all of it, but its planes are
// written and accumulated in equal parts of at most this many pairs (the parts' FP64 adds are
// the only difference from one pass). The parts depend on the slab's own length only, so a
// slab gives the same bits in whatever call it lies.
//   * With more tiles per frequency than SMs, a round of CTAs reads a frequency's planes
//     while the rest of its tiles wait for the next round: the planes come from L2 again
//     only if they (3 digits x R rows x pairs) leave room there. Measured at 1200 columns,
//     full calls of a million pairs, one kernel: 739-747 TFLOP/s with 8192 and 12288 pairs
//     (60 and 90 MB), 718-723 with 16384 (120 MB), 641 with 32768.
//   * Otherwise a round's CTAs walk the same pairs together: the whole slab.
static int64_t split_part_most(int64_t slab, int ntile, int64_t R) {
  if (ntile <= SP_SMS) return slab;
  return std::min<int64_t>(slab, std::max<int64_t>(4096, (90ll << 20) / (SP_SF * R) / SP_KB * SP_KB));
}

// slab: band pairs per exact int32 slab, a multiple of SP_KB in [SP_KB, SP_SLAB]; R plane rows.
// Two operand buffers when there is more than one part: the next part is quantized
// while one accumulates. The size never falls with P, so scratch for a call holds every
// shorter one of its width: the planes of one slab take the slab's pairs at most (two parts
// share them), those of several slabs two of the longest parts.
static SplitLayout split_layout_of(int64_t P, int nblk, int64_t R, int ntile, int ncol, int nw, int slab) {
  SplitLayout L;
  L.Ps = std::min<int64_t>((int64_t)align_up((size_t)std::max<int64_t>(P, 1), SP_KB), slab);
  L.most = split_part_most(slab, ntile, R);
  L.pairs = P > slab ? 2 * L.most : std::min(L.Ps, 2 * L.most);
  L.nblk = nblk;
  L.R = R;
  L.nstat = P > slab ? 2 : 1;
  L.f_bytes = align_up((size_t)SP_SLOT * nw * R * L.pairs, 1024);
  L.g_bytes = align_up(sizeof(double) * (size_t)nw * L.Ps, 256);
  L.s_bytes = align_up(sizeof(double) * (size_t)std::max(ncol, 1), 256);
  L.w_bytes = align_up(sizeof(double) * (size_t)std::max(nw, 1), 256);
  L.sg_bytes = align_up(sizeof(int) * (size_t)std::max(nw, 1), 256);
  return L;
}

static SplitLayout split_layout(int64_t P, int N, int nw, int slab) {
  const int nblk = (N + SP_TILE - 1) / SP_TILE;
  // an even number of 64-blocks, so a CTA pair's second A tile always exists
  return split_layout_of(P, nblk, (int64_t)((nblk + 1) / 2 * 2) * SP_ROWS, split_ntile(N, SP_WIDE_BN, nblk), N, nw,
                         slab);
}

static int clamp_slab(int slab) {
  if (slab <= 0) return SP_SLAB;
  return (int)std::min<int64_t>(SP_SLAB, std::max<int64_t>(SP_KB, slab / SP_KB * SP_KB));
}

size_t split_workspace_bytes(int64_t P, int N, int nw, int slab) {
  slab = clamp_slab(slab);
  return split_layout(P, N, nw, slab).bytes();
}
// Bytes that hold the partial tiles of any call: two per CTA.
size_t split_part_bytes(int num_sms, bool real) {
  return align_up(sizeof(double) * 2 * (size_t)num_sms * split_part_elems(real, SP_WIDE_BN), 256);
}

size_t split_workspace_bytes(int64_t P, int N, int nw) {
  return split_workspace_bytes(P, N, nw, SP_SLAB);
}

void timing_mark(spx_ctx* ctx, cudaStream_t s, int kind);

// Launches the one-CTA kernel for one slab (prm.nitems, nk and the operands set), with the
// last items cut over all CTAs when that pays and `part` has room for the partial tiles.
template <bool REAL, int BN>
static int split_gram_launch(spx_ctx* ctx, const CUtensorMap& mapA, const CUtensorMap& mapB, SplitParams prm,
                             double* part, cudaStream_t stream, bool chained, int* launches) {
  const size_t smem = sizeof(SplitSmemT<2 * BN>) + 1024;
  int rc = check_cuda(ctx, cudaFuncSetAttribute(split_gram_kernel<REAL, BN>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                      "split_gram_kernel attribute");
  if (rc) return rc;
  prm.ncut = part ? split_cut_ctas(prm.nitems, prm.nk, ctx->num_sms, REAL) : 0;
  prm.whole = prm.ncut ? prm.nitems / ctx->num_sms * ctx->num_sms : prm.nitems;
  prm.part = prm.ncut ? part : nullptr;
  const int grid = std::min(prm.whole ? prm.whole : prm.ncut, ctx->num_sms);
  if ((rc = check_cuda(ctx, launch_chained(split_gram_kernel<REAL, BN>, grid, SP1_THREADS, smem, stream, chained, mapA,
                                           mapB, prm),
                       "split_gram_kernel launch")))
    return rc;
  *launches += 1;
  if (prm.ncut) {
    const int ny = (REAL ? 2 : 1) * BN * 4 / SP1_EPI / split_finish_step<REAL>();
    if ((rc = check_cuda(ctx, launch_chained(split_gram_finish_kernel<REAL, BN>, dim3(prm.ncut - 1, ny), 32 * SP1_EPI, 0,
                                             stream, true, prm, grid),
                         "split_gram_finish_kernel launch")))
      return rc;
    *launches += 1;
  }
  return SPX_OK;
}

// The buffers of a call: `n` operand buffers of Pp[b] pairs each, and the statistics of the
// slabs in turn.
struct SplitBuf {
  int8_t* F;
  int64_t Pp;
  double *G, *sA, *wmax;
  int* wsgn;
};
static int split_buffers(const SplitLayout& L, int64_t P, int nw, uint8_t* base, SplitBuf (&buf)[2]) {
  const int64_t rest = P % L.Ps, p0 = std::max(L.part(L.Ps), rest ? L.part(rest) : 0);
  buf[0].Pp = p0;
  buf[1].Pp = L.nstat == 1 ? std::min(p0, L.Ps - p0) : p0;   // one slab: what its first part leaves
  buf[0].F = (int8_t*)base;
  buf[1].F = (int8_t*)base + (size_t)SP_SLOT * nw * L.R * p0;
  for (int b = 0; b < 2; ++b) {
    uint8_t* s0 = base + L.f_bytes + (b < L.nstat ? b : 0) * (L.g_bytes + L.s_bytes + L.w_bytes + L.sg_bytes);
    buf[b].G = (double*)s0;
    buf[b].sA = (double*)(s0 + L.g_bytes);
    buf[b].wmax = (double*)(s0 + L.g_bytes + L.s_bytes);
    buf[b].wsgn = (int*)(s0 + L.g_bytes + L.s_bytes + L.w_bytes);
  }
  return buf[1].Pp > 0 ? 2 : 1;
}

// One part of a slab: slab pairs [p0, p0 + len), part [off, off + plen) of them.
struct SplitStep {
  int64_t p0;
  int len, off, plen;
  int sb, b;   // buffer of the slab's statistics, of the part's planes
  bool last;   // nothing is prepared beside this part's accumulation
};

// Runs the parts of a call: stat(step, stream) before a slab's first part, then
// quant(step, stream), on the preparation stream, one part ahead of gram(step) on `stream`. A
// single part has nothing to run beside and stays on `stream`. The statistics buffer of
// slab s is reused by slab s + 2, whose first part waits for a part of slab s + 1 at least.
template <class Stat, class Quant, class Gram>
static int split_run_steps(spx_ctx* ctx, const SplitLayout& L, int64_t P, int nbuf, cudaStream_t stream, Stat stat,
                           Quant quant, Gram gram) {
  std::vector<SplitStep> steps;
  for (int64_t p0 = 0, s = 0; p0 < P; p0 += L.Ps, ++s) {
    const int len = (int)std::min<int64_t>(L.Ps, P - p0), part = (int)L.part(len);
    for (int off = 0; off < len; off += part)
      steps.push_back({p0, len, off, std::min(part, len - off), (int)(s % L.nstat), (int)(steps.size() % nbuf), false});
  }
  steps.back().last = true;
  const bool two = nbuf == 2;   // the kernels of a part lie on two streams, unchained
  cudaStream_t ps = two ? ctx->prep_stream : stream;
  cudaEvent_t prep_done[2] = {ctx->sev[1], ctx->sev[2]};
  cudaEvent_t gram_done[2] = {ctx->sev[3], ctx->sev[4]};
  int rc = SPX_OK;
  auto prep = [&](const SplitStep& t) -> int {
    if (t.off == 0 && (rc = stat(t, ps))) return rc;
    if ((rc = quant(t, ps))) return rc;
    return two ? check_cuda(ctx, cudaEventRecord(prep_done[t.b], ps), "event") : SPX_OK;
  };
  // the preparation stream starts after everything already queued on `stream` (whatever
  // produced cprod and the weights, and the last call's use of the buffers)
  if (two && ((rc = check_cuda(ctx, cudaEventRecord(ctx->sev[0], stream), "event")) ||
              (rc = check_cuda(ctx, cudaStreamWaitEvent(ps, ctx->sev[0], 0), "event"))))
    return rc;
  timing_mark(ctx, stream, 0);
  if ((rc = prep(steps[0]))) return rc;
  for (size_t k = 0; k < steps.size(); ++k) {
    const SplitStep& t = steps[k];
    if (two && (rc = check_cuda(ctx, cudaStreamWaitEvent(stream, prep_done[t.b], 0), "event"))) return rc;
    timing_mark(ctx, stream, 1);
    if ((rc = gram(t))) return rc;
    timing_mark(ctx, stream, 2);  // the accumulation interval ends with the kernel
    if (two && (rc = check_cuda(ctx, cudaEventRecord(gram_done[t.b], stream), "event"))) return rc;
    if (k + 1 < steps.size()) {
      // the next part goes into the buffer that part k - 1 accumulated from
      if (k >= 1 && (rc = check_cuda(ctx, cudaStreamWaitEvent(ps, gram_done[steps[k + 1].b], 0), "event")))
        return rc;
      if ((rc = prep(steps[k + 1]))) return rc;
    }
  }
  return SPX_OK;
}

// variant: 1 one CTA per 64 x 64 tile, 2 CTA pair, 5 one CTA per 64 x 80 tile, 0 the
// context's choice; slab: pairs per exact int32 slab (0 = 32768); part: split_part_bytes for
// partial tiles, or NULL.
static int split_chi0_run(spx_ctx* ctx, const double2* M, int64_t ldc, int64_t P, int N, const SplitStat& src,
                          int nw, double2* out, void* ws, size_t ws_bytes, double* part, cudaStream_t stream,
                          int* launches, int variant, int slab) {
  if (P <= 0 || N <= 0 || nw <= 0) return SPX_OK;
  slab = clamp_slab(slab);
  SplitLayout L = split_layout(P, N, nw, slab);
  if (!ws || ws_bytes < split_workspace_bytes(P, N, nw, slab))
    return set_error(ctx, SPX_EINVAL, "split workspace too small");
  uint8_t* base = (uint8_t*)align_up((size_t)ws, 1024);
  SplitBuf buf[2];
  const int nbuf = split_buffers(L, P, nw, base, buf);

  // planes in HBM: [plane][k-block][row][K bytes]; TMA dims (K, row, k-block, plane)
  // with increasing strides; a box (K, rows, 1, 3 planes) lands as [plane][row][K]
  if (variant == 0) variant = ctx->opt.split_variant;
  if (variant == 0)   // untuned: one CTA per tile
    variant = split_wide(N, L.nblk, nw, buf[0].Pp / SP_KB, ctx->num_sms, false, part && nbuf == 1) ? 5 : 1;
  const bool pair = variant == 2;
  const bool wide = variant == 5;                  // one CTA per 64 x 80 tile (N = 160)
  // only the CTA pair needs an even number of 64-column blocks in the planes (the
  // buffers are sized for it either way)
  if (!pair) L.R = (int64_t)L.nblk * SP_ROWS;
  CUtensorMap mapF[2], mapFh[2], mapW[2];
  for (int b = 0; b < nbuf; ++b) {
    const uint64_t nkb = (uint64_t)(buf[b].Pp / SP_KB);
    const uint64_t st[3] = {SP_KB, (uint64_t)L.R * SP_KB, nkb * L.R * SP_KB};
    const uint64_t d[4] = {SP_KB, (uint64_t)L.R, nkb, (uint64_t)SP_SLOT * nw};
    const uint32_t bx[4] = {SP_KB, SP_ROWS, 1, SP_SF};
    int rc0 = make_tmap_u8_4d(ctx, &mapF[b], buf[b].F, d, st, bx, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc0) return rc0;
    const uint32_t bh[4] = {SP_KB, SP2_BROWS, 1, SP_SF};
    rc0 = make_tmap_u8_4d(ctx, &mapFh[b], buf[b].F, d, st, bh, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc0) return rc0;
    const uint32_t bw[4] = {SP_KB, 2 * SP_WIDE_BN, 1, SP_SF};
    rc0 = make_tmap_u8_4d(ctx, &mapW[b], buf[b].F, d, st, bw, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc0) return rc0;
  }
  int rc = SPX_OK;

  const size_t smem2 = sizeof(Split2Smem) + 1024;
  if (pair) cudaFuncSetAttribute(split_gram2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
  const int nbr = (N + SP_TILE - 1) / SP_TILE;
  int ntile2 = 0;
  for (int bj = 0; bj < L.nblk; ++bj) ntile2 += bj / 2 + 1;
  const int ntile_used = pair ? ntile2 : split_ntile(N, wide ? SP_WIDE_BN : SP_TILE, nbr);
  const int nitems = ntile_used * nw;
  const int npad = (int)(L.R / 2);  // columns covered by the stacked rows
  // CTA-pair launch: as many clusters as can be resident at once (persistent)
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute cattr[1];
  int nclusters = 0;
  if (pair) {
    cattr[0].id = cudaLaunchAttributeClusterDimension;
    cattr[0].val.clusterDim.x = 2;
    cattr[0].val.clusterDim.y = 1;
    cattr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(SP_THREADS);
    cfg.dynamicSmemBytes = smem2;
    cfg.stream = stream;
    cfg.attrs = cattr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(2 * (ctx->num_sms / 2));
    int maxc = 0;
    rc = check_cuda(ctx, cudaOccupancyMaxActiveClusters(&maxc, split_gram2_kernel, &cfg),
                    "cudaOccupancyMaxActiveClusters");
    if (rc) return rc;
    if (maxc <= 0) return set_error(ctx, SPX_ENOTSUP, "no CTA-pair cluster fits on this device");
    nclusters = std::min(nitems, maxc);
    cfg.gridDim = dim3(2 * nclusters);
  }

  auto stat = [&](const SplitStep& t, cudaStream_t ps) -> int {
    const int ncol = (int)align_up((size_t)N, SPS_CL);
    split_stat_kernel<false><<<ncol + nw * SPS_CL, SPS_THREADS, 0, ps>>>(
        reinterpret_cast<const double*>(M), ldc, t.p0, t.len, (int)align_up((size_t)t.len, SP_KB), N, ncol, src,
        buf[t.sb].sA, buf[t.sb].wmax, buf[t.sb].wsgn, buf[t.sb].G);
    ++*launches;
    return check_cuda(ctx, cudaGetLastError(), "split_stat_kernel launch");
  };
  auto quant = [&](const SplitStep& t, cudaStream_t ps) -> int {
    const int nchunk = (int)align_up((size_t)t.plen, SP_KB) / 16;  // 16-pair chunks; npad is a multiple of 64
    const int64_t nthr = (int64_t)npad * nchunk * 2;                // 8-pair tasks
    ++*launches;
    return check_cuda(ctx, launch_chained(split_quantize_kernel, (unsigned)((nthr + 127) / 128), 128, 0, ps, nbuf == 1,
                                          M, ldc, t.p0 + t.off, t.plen, nchunk, N, npad, L.R, buf[t.b].Pp, nw, buf[t.sb].sA,
                                          buf[t.sb].wsgn, buf[t.sb].G + t.off, (int)align_up((size_t)t.len, SP_KB),
                                          buf[t.b].F),
                      "split_quantize_kernel launch");
  };
  auto gram = [&](const SplitStep& t) -> int {
    SplitParams prm;
    prm.N = N;
    prm.nbr = nbr;
    prm.ntile = ntile_used;
    prm.nw = nw;
    prm.nitems = nitems;
    prm.nk = (int)align_up((size_t)t.plen, SP_KB) / SP_KB;
    prm.sA = buf[t.sb].sA;
    prm.wmax = buf[t.sb].wmax;
    prm.wsgn = buf[t.sb].wsgn;
    prm.out = reinterpret_cast<double*>(out);
    prm.npack = (int64_t)N * (N + 1) / 2;
    prm.status = ctx->d_status;
    prm.timeout_ns =
        (uint64_t)(ctx->opt.timeout_ms > 0 ? ctx->opt.timeout_ms : 4000) * 1000000ull;
    if (pair) {
      ++*launches;
      return check_cuda(ctx, cudaLaunchKernelEx(&cfg, split_gram2_kernel, mapF[t.b], mapFh[t.b], prm),
                        "split_gram2_kernel launch");
    }
    if (wide) return split_gram_launch<false, SP_WIDE_BN>(ctx, mapF[t.b], mapW[t.b], prm, t.last ? part : nullptr, stream, nbuf == 1, launches);
    return split_gram_launch<false, SP_TILE>(ctx, mapF[t.b], mapF[t.b], prm, t.last ? part : nullptr, stream, nbuf == 1, launches);
  };
  return split_run_steps(ctx, L, P, nbuf, stream, stat, quant, gram);
}

// The accumulation with given weights W (ldw, nw).
int split_chi0_slab(spx_ctx* ctx, const double2* M, int64_t ldc, int64_t P, int N, const double* W,
                    int64_t ldw, int nw, double2* out, void* ws, size_t ws_bytes, void* part,
                    cudaStream_t stream, int* launches, int variant, int slab) {
  return split_chi0_run(ctx, M, ldc, P, N, SplitStat{W, ldw, nullptr, nullptr, 0.0, nullptr}, nw, out, ws,
                        ws_bytes, (double*)part, stream, launches, variant, slab);
}

// The accumulation with the HILBERT NONE weights of ediff (the same bits as K6's).
int split_chi0_ediff(spx_ctx* ctx, const double2* M, int64_t ldc, int64_t P, int N, const double* ediff,
                     const double* wscale, double scale_all, int nw, const double* omega, double2* out,
                     void* ws, size_t ws_bytes, void* part, cudaStream_t stream, int* launches, int variant,
                     int slab) {
  return split_chi0_run(ctx, M, ldc, P, N, SplitStat{nullptr, 0, ediff, wscale, scale_all, omega}, nw, out, ws,
                        ws_bytes, (double*)part, stream, launches, variant, slab);
}

// Real layout: 128 columns per block, one plane row per column.
static SplitLayout split_layout_real(int64_t P, int N, int nw) {
  const int nblk = (N + SP_ROWS - 1) / SP_ROWS;
  return split_layout_of(P, nblk, (int64_t)nblk * SP_ROWS, split_ntile((N + 1) / 2, SP_WIDE_BN, nblk), N, nw, SP_SLAB);
}

size_t split_workspace_bytes_real(int64_t P, int N, int nw) { return split_layout_real(P, N, nw).bytes(); }

// The -DINV accumulation (src/susceptibility.f:1197, re(k) = cprod(k,i) * cprod(k,j)):
// real M (ldc, N), real packed out (npack, nw), the folded 6-product int8 contraction
// on 128 x 160 real tiles (N = 160 MMAs) or 128 x 128 (when those take less time, or the
// context's split variant is 1), one CTA per tile. HILBERT NONE weights of ediff.
int split_chi0_real_ediff(spx_ctx* ctx, const double* M, int64_t ldc, int64_t P, int N, const double* ediff,
                          const double* wscale, double scale_all, int nw, const double* omega, double* out,
                          void* ws, size_t ws_bytes, cudaStream_t stream, int* launches) {
  if (P <= 0 || N <= 0 || nw <= 0) return SPX_OK;
  const SplitStat src{nullptr, 0, ediff, wscale, scale_all, omega};
  const SplitLayout L = split_layout_real(P, N, nw);
  if (!ws || ws_bytes < L.bytes()) return set_error(ctx, SPX_EINVAL, "split workspace too small");
  uint8_t* base = (uint8_t*)align_up((size_t)ws, 1024);
  SplitBuf buf[2];
  const int nbuf = split_buffers(L, P, nw, base, buf);
  double* part = (double*)ctx->part;   // partial tiles
  const bool wide = ctx->opt.split_variant != 1 && (ctx->opt.split_variant != 0 || split_wide((N + 1) / 2, L.nblk, nw, buf[0].Pp / SP_KB,
                                                                                       ctx->num_sms, true, part && nbuf == 1));
  CUtensorMap mapF[2], mapW[2];
  for (int b = 0; b < nbuf; ++b) {
    const uint64_t nkb = (uint64_t)(buf[b].Pp / SP_KB);
    const uint64_t st[3] = {SP_KB, (uint64_t)L.R * SP_KB, nkb * L.R * SP_KB};
    const uint64_t d[4] = {SP_KB, (uint64_t)L.R, nkb, (uint64_t)SP_SLOT * nw};
    const uint32_t bx[4] = {SP_KB, SP_ROWS, 1, SP_SF};
    int rc0 = make_tmap_u8_4d(ctx, &mapF[b], buf[b].F, d, st, bx, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc0) return rc0;
    const uint32_t bw[4] = {SP_KB, 2 * SP_WIDE_BN, 1, SP_SF};
    rc0 = make_tmap_u8_4d(ctx, &mapW[b], buf[b].F, d, st, bw, CU_TENSOR_MAP_SWIZZLE_64B);
    if (rc0) return rc0;
  }
  // tiles in 128-row blocks of the real rows; wide tiles in 160-column blocks
  const int nbr = L.nblk;
  const int ntile = split_ntile((N + 1) / 2, wide ? SP_WIDE_BN : SP_TILE, nbr);
  const int nitems = ntile * nw;
  const int npad = (int)L.R;
  auto stat = [&](const SplitStep& t, cudaStream_t ps) -> int {
    const int ncol = (int)align_up((size_t)N, SPS_CL);
    split_stat_kernel<true><<<ncol + nw * SPS_CL, SPS_THREADS, 0, ps>>>(
        M, ldc, t.p0, t.len, (int)align_up((size_t)t.len, SP_KB), N, ncol, src, buf[t.sb].sA, buf[t.sb].wmax,
        buf[t.sb].wsgn, buf[t.sb].G);
    ++*launches;
    return check_cuda(ctx, cudaGetLastError(), "split_stat_kernel (real) launch");
  };
  auto quant = [&](const SplitStep& t, cudaStream_t ps) -> int {
    const int nchunk = (int)align_up((size_t)t.plen, SP_KB) / 16;
    // npad columns (a multiple of 128) x 16-pair chunks, 128 threads a block
    ++*launches;
    return check_cuda(ctx, launch_chained(split_quantize_real_kernel, (unsigned)((int64_t)npad * nchunk / 128), 128, 0, ps,
                                          nbuf == 1, M, ldc, t.p0 + t.off, t.plen, nchunk, N, npad, L.R, buf[t.b].Pp, nw,
                                          buf[t.sb].sA, buf[t.sb].wsgn, buf[t.sb].G + t.off,
                                          (int)align_up((size_t)t.len, SP_KB), buf[t.b].F),
                      "split_quantize_real_kernel launch");
  };
  auto gram = [&](const SplitStep& t) -> int {
    SplitParams prm;
    prm.N = N;
    prm.nbr = nbr;
    prm.ntile = ntile;
    prm.nw = nw;
    prm.nitems = nitems;
    prm.nk = (int)align_up((size_t)t.plen, SP_KB) / SP_KB;
    prm.sA = buf[t.sb].sA;
    prm.wmax = buf[t.sb].wmax;
    prm.wsgn = buf[t.sb].wsgn;
    prm.out = out;
    prm.npack = (int64_t)N * (N + 1) / 2;
    prm.status = ctx->d_status;
    prm.timeout_ns = (uint64_t)(ctx->opt.timeout_ms > 0 ? ctx->opt.timeout_ms : 4000) * 1000000ull;
    if (wide) return split_gram_launch<true, SP_WIDE_BN>(ctx, mapF[t.b], mapW[t.b], prm, t.last ? part : nullptr, stream, nbuf == 1, launches);
    return split_gram_launch<true, SP_TILE>(ctx, mapF[t.b], mapF[t.b], prm, t.last ? part : nullptr, stream, nbuf == 1, launches);
  };
  return split_run_steps(ctx, L, P, nbuf, stream, stat, quant, gram);
}

}  // namespace spx

// ---------------------------------------------------------------------------
// K4s: the interstitial product GEMM of the explicit convolution
// (src/wavefproducts.f:945, cprod += conj(cpw2^H cpw3)/sqrt(vol)) on the same
// int8 digit slices as K2. C_b(m, col) = alpha * sum_k A_b(m, k) conj(B_b(col, k)):
// A = the unoccupied coefficients (rows n'), B = the gathered convolution
// cpw0(G2 - G_M + g) (rows (n, ig)), one batch per k point. Each row is scaled
// by its own largest |Re|, |Im| over k; A keeps 3 digits, B 4, and the nine
// products with t + u <= 3 are summed exactly in int32 (k <= 32768 per launch),
// so the only rounding is the slicing: 2^-17/127 of A's row scale per value, so
// |error of C(m, col)| <= 2^-17/127 * crest(A_m) * ||A_m|| ||B_col||.
// Items are rectangular (batch, column tile, row tile) of 64 x 64 complex values, row tiles
// fastest so that concurrent CTAs share the large B tile through L2. Both operands use K2's
// interleaved rows, so the fragments of a row's two parts meet in neighbouring lanes and a
// warp's values of one column are 256 contiguous bytes of cprod.
namespace spx {

struct SgParams {
  int nbatch, mtiles, ntiles, nitems, nk;
  int64_t RA, RB;          // real-stacked rows per batch of the A and B planes
  int M, ncol, ncin;       // valid rows of A, columns (= rows of B), col = n*ncin + c
  const double* sA;        // row scales [batch][mtiles*64]
  const double* sB;        // [batch][ntiles*64]
  double* out;             // cprod as doubles, at (row 0, column 0) of batch 0
  int64_t sO2, sOn, sOc;   // complex strides: batch, n, c
  double alpha;
  int overwrite;           // 1: store (the output range holds nothing yet), 0: add
  int* status;
  uint64_t timeout_ns;
};

// One CTA per tile: MMAs of N = 128 (an MMA of N = 64 takes the same time, bound by the
// instruction rate: 32-column tiles with two TMEM buffers took 40 ms of the 27 x 300 x 40560 x
// 3000 products, this form 24 ms). The four orders of 128 columns fill TMEM, so the next
// tile's MMAs wait while eight epilogue warps read it into registers (about 3 % of a tile's 47
// stages); scaling and stores run beside them.
constexpr int SG_ST = 4;

struct __align__(1024) SgSmem {
  uint8_t a[SG_ST][SP_SA][SP_PLANE];
  uint8_t b[SG_ST][SP_SB][SP_PLANE];
  uint64_t full[SG_ST];
  uint64_t empty[SG_ST];
  uint64_t tfull, tempty, mdone;
  uint32_t tmem_base;
};

// T = ((D0*256 + D1)*256 + D2)*256 + D3 for 16 columns, orders 128 columns apart.
__device__ __forceinline__ void load_orders16(uint32_t taddr, long long (&T)[16]) {
  int32_t r[4][16];
  __syncwarp();   // the read is warp-wide; lanes of rows past the end skip the stores before it
#pragma unroll
  for (int g = 0; g < 4; ++g) tmem_ld16(taddr + (uint32_t)(g * SP_ROWS), r[g]);
  tmem_wait_ld();
#pragma unroll
  for (int k = 0; k < 16; ++k)
    T[k] = (((long long)r[0][k] * 256 + r[1][k]) * 256 + r[2][k]) * 256 + r[3][k];
}

__global__ void __launch_bounds__(SP1_THREADS, 1)
    split_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                      SgParams prm) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  SgSmem& sm = *reinterpret_cast<SgSmem*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < SG_ST; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    mbar_init(&sm.tfull, 1);
    mbar_init(&sm.tempty, SP1_EPI);
    mbar_init(&sm.mdone, 1);
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(&sm.tmem_base, SP_TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  const int mtiles = prm.mtiles, ntiles = prm.ntiles;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 0;
      bool issued[SG_ST];
      uint32_t last_ph[SG_ST];
      for (int s = 0; s < SG_ST; ++s) issued[s] = false, last_ph[s] = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < prm.nitems && ok; item += gridDim.x) {
        const int mt = item % mtiles, r = item / mtiles, ct = r % ntiles, b = r / ntiles;
        const int ra = (int)(b * prm.RA) + mt * SP_ROWS, rb = (int)(b * prm.RB) + ct * SP_ROWS;
        for (int ks = 0; ks < prm.nk; ++ks) {
          if (!mbar_wait(&sm.empty[st], ph ^ 1u, prm.timeout_ns, prm.status)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&sm.full[st], (uint32_t)((SP_SA + SP_SB) * SP_PLANE));
          tma_load_4d(&sm.a[st][0][0], &mapA, 0, ra, ks, 0, &sm.full[st]);
          tma_load_4d(&sm.b[st][0][0], &mapB, 0, rb, ks, 0, &sm.full[st]);
          issued[st] = true;
          last_ph[st] = ph;
          if (++st == SG_ST) st = 0, ph ^= 1u;
        }
      }
      for (int s = 0; s < SG_ST; ++s)
        if (issued[s]) mbar_drain(&sm.full[s], last_ph[s], prm.timeout_ns);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int st = 0;
      uint32_t ph = 0;
      int j = 0;
      bool committed = false;
      for (int item = blockIdx.x; item < prm.nitems; item += gridDim.x, ++j) {
        // the previous item's accumulators have been read (first item: immediately)
        if (!mbar_wait(&sm.tempty, (uint32_t)(j & 1) ^ 1u, prm.timeout_ns, prm.status)) break;
        tc_fence_after();
        bool ok = true;
        for (int ks = 0; ks < prm.nk; ++ks) {
          if (!mbar_wait(&sm.full[st], ph, prm.timeout_ns, prm.status)) {
            ok = false;
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < SP_NKS; ++kk) {
            uint64_t da[SP_SA], db[SP_SB];
#pragma unroll
            for (int t = 0; t < SP_SA; ++t) da[t] = desc_sw64(&sm.a[st][t][0]) + (uint64_t)(kk * 2);
#pragma unroll
            for (int u = 0; u < SP_SB; ++u) db[u] = desc_sw64(&sm.b[st][u][0]) + (uint64_t)(kk * 2);
            const uint32_t k0 = (ks > 0 || kk > 0);
            mma_i8<1>(tmem + 0 * SP_ROWS, da[0], db[0], SP_IDESC, k0);
            mma_i8<2>(tmem + 1 * SP_ROWS, da[0], db[1], SP_IDESC, k0);
            mma_i8<2>(tmem + 2 * SP_ROWS, da[0], db[2], SP_IDESC, k0);
            mma_i8<3>(tmem + 3 * SP_ROWS, da[0], db[3], SP_IDESC, k0);
            mma_i8<1>(tmem + 1 * SP_ROWS, da[1], db[0], SP_IDESC, 1u);
            mma_i8<2>(tmem + 2 * SP_ROWS, da[1], db[1], SP_IDESC, 1u);
            mma_i8<3>(tmem + 3 * SP_ROWS, da[1], db[2], SP_IDESC, 1u);
            mma_i8<1>(tmem + 2 * SP_ROWS, da[2], db[0], SP_IDESC, 1u);
            mma_i8<3>(tmem + 3 * SP_ROWS, da[2], db[1], SP_IDESC, 1u);
          }
          tc_commit(&sm.empty[st]);
          committed = true;
          if (++st == SG_ST) st = 0, ph ^= 1u;
        }
        if (!ok) break;
        tc_commit(&sm.tfull);
      }
      if (committed) {
        tc_commit(&sm.mdone);
        mbar_drain(&sm.mdone, 0u, prm.timeout_ns);
      }
    }
  } else {
    // ---- epilogue: two warps per TMEM lane quarter, 32 complex columns each ----
    const int q = warp & 3, h = (warp - 2) >> 2, c = lane & 1;
    const uint32_t tl = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(SP_TILE * h);
    int j = 0;
    for (int item = blockIdx.x; item < prm.nitems; item += gridDim.x, ++j) {
      if (!mbar_wait_idle(&sm.tfull, (uint32_t)(j & 1), prm.timeout_ns, prm.status)) break;
      tc_fence_after();
      const int mt = item % mtiles, r = item / mtiles, ct = r % ntiles, b = r / ntiles;
      long long o[SP_TILE / 2];
#pragma unroll
      for (int cc = 0; cc < SP_TILE / 16; ++cc) {
        long long T[16];
        load_orders16(tl + (uint32_t)(16 * cc), T);
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          // A conj(B): re = ArBr + AiBi (even lanes), im = AiBr - ArBi
          const long long pb = __shfl_xor_sync(0xffffffffu, T[2 * jj + 1], 1);
          o[8 * cc + jj] = c == 0 ? T[2 * jj] + pb : T[2 * jj] - pb;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.tempty);
      const int gm = mt * SP_TILE + 16 * q + lane / 2;
      if (gm >= prm.M) continue;
      const double fac = prm.alpha * prm.sA[(int64_t)b * mtiles * SP_TILE + gm] *
                         (1.0 / (127.0 * 127.0 * 16777216.0));
      const int gc0 = ct * SP_TILE + 32 * h;
      const double* sbb = prm.sB + (int64_t)b * ntiles * SP_TILE + gc0;
      int n = gc0 / prm.ncin, cin = gc0 - n * prm.ncin;
      double* ob = prm.out + 2 * (b * prm.sO2 + gm) + c;
#pragma unroll
      for (int k = 0; k < SP_TILE / 2; ++k) {
        if (gc0 + k >= prm.ncol) break;
        double* oc = ob + 2 * (n * prm.sOn + cin * prm.sOc);
        const double v = fac * sbb[k] * (double)o[k];
        *oc = prm.overwrite ? v : *oc + v;
        if (++cin == prm.ncin) cin = 0, ++n;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, SP_TMEM_COLS);
}

// Row sources of the two operands, k running through the caller's order of the plane
// waves (the box order of their G vectors, so that a row's gather walks the convolved grid
// upwards; the integer sums do not depend on it): A rows of cpw, B rows of the grid.
struct SgSrcRows {
  const double2* base;
  int64_t ld, bstride;
  const int* kperm;         // plane wave of the k-th position
  __device__ __forceinline__ double2 get(int b, int r, int k) const {
    return __ldg(base + b * bstride + (int64_t)r * ld + kperm[k]);
  }
};
struct SgSrcGather {
  const double2* grid;      // [batch][n][box]
  int64_t bstride, nstride;
  const int64_t* coff;      // per c
  const int* koff;          // per position k
  int ncin;
  __device__ __forceinline__ double2 get(int b, int r, int k) const {
    const int n = r / ncin, c = r - n * ncin;
    return __ldg(grid + b * bstride + n * nstride + coff[c] + koff[k]);
  }
};

// One CTA per row of up to SGP_K values: the row's scale max_k max(|Re|, |Im|) (0 for padding
// rows) and its S digits in one pass over its (gathered) values, kept in registers between.
// A thread holds four runs of four consecutive k; planes [t][k-block][row][64 B] as below.
// Bound by the gather through L2 (53 GB in 16-byte pieces for the 27 x 40560 rows of 3000):
// 17 ms, against 26 ms as a pass for the scales and one for the digits, plane waves in the
// caller's order.
constexpr int SGP_T = 256, SGP_K = 16 * SGP_T;
template <int S, class Src>
__global__ void __launch_bounds__(SGP_T)
    sgemm_prep_kernel(Src src, int rows, int rows_pad, int K, int nkb, int nbatch, int64_t R,
                      double* __restrict__ s, int8_t* __restrict__ planes) {
  __shared__ double red[SGP_T / 32];
  const int r = blockIdx.x, b = blockIdx.y;
  double2 v[16];
  double m = 0.0;
#pragma unroll
  for (int e = 0; e < 16; ++e) {
    const int k = 4 * (threadIdx.x + SGP_T * (e >> 2)) + (e & 3);
    v[e] = r < rows && k < K ? src.get(b, r, k) : make_double2(0.0, 0.0);
    m = fmax(m, fmax(fabs(v[e].x), fabs(v[e].y)));
  }
  m = block_max(m, red);
  if (threadIdx.x == 0) s[(int64_t)b * rows_pad + r] = m;
  const double inv = m > 0.0 ? 127.0 * (S == 4 ? 16777216.0 : 65536.0) / m : 0.0;
  const int64_t rows_total = (int64_t)nbatch * R;
  const int64_t pstride = (int64_t)nkb * rows_total * SP_KB;
  const int64_t row = ((int64_t)b * R + split_row_re(r)) * SP_KB;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = 4 * (threadIdx.x + SGP_T * q);
    if (k >= nkb * SP_KB) break;
    uint32_t yr[4], yi[4], pr[S], pi[S];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      yr[e] = round_mul(v[4 * q + e].x, inv);
      yi[e] = round_mul(v[4 * q + e].y, inv);
    }
    digit_planes<S>(yr, pr);
    digit_planes<S>(yi, pi);
    const int64_t o = (int64_t)(k / SP_KB) * rows_total * SP_KB + row + k % SP_KB;
#pragma unroll
    for (int t = 0; t < S; ++t) {
      *reinterpret_cast<uint32_t*>(planes + o + t * pstride) = pr[t];
      *reinterpret_cast<uint32_t*>(planes + o + SP_KB + t * pstride) = pi[t];
    }
  }
}

// Longer rows take two passes:
// s[b*rows_pad + r] = max_k max(|Re|, |Im|) of row r of batch b (0 for padding rows).
template <class Src>
__global__ void sgemm_rowmax_kernel(Src src, int rows, int rows_pad, int K, double* s) {
  const int r = blockIdx.x, b = blockIdx.y;
  double m = 0.0;
  if (r < rows)
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
      const double2 v = src.get(b, r, k);
      m = fmax(m, fmax(fabs(v.x), fabs(v.y)));
    }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) s[(int64_t)b * rows_pad + r] = m;
  }
}

// S digits of round(x * 127/s * 2^(8(S-1))) into planes [t][k-block][row][64 B] with K2's
// interleaved rows (split_row_re). One thread = one row and 16 consecutive k; a warp = 8
// consecutive rows x the 4 quarters of a k-block.
template <int S, class Src>
__global__ void __launch_bounds__(128)
    sgemm_quant_kernel(Src src, int rows, int rows_pad, int K, int nkb, int nbatch, int64_t R,
                       const double* __restrict__ s, int8_t* __restrict__ planes) {
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int ngroup = rows_pad / 8;
  if (tid >= (int64_t)ngroup * 32 * nkb * nbatch) return;
  const int lane8 = (int)(tid & 7), quarter = (int)((tid >> 3) & 3);
  const int64_t rest = tid >> 5;
  const int r = (int)(rest % ngroup) * 8 + lane8;
  const int64_t kbb = rest / ngroup;
  const int kb = (int)(kbb % nkb), b = (int)(kbb / nkb);
  const int k0 = kb * SP_KB + quarter * 16;
  const int64_t rows_total = (int64_t)nbatch * R;
  const int64_t rr = (int64_t)b * R + split_row_re(r);
  const int64_t pstride = (int64_t)nkb * rows_total * SP_KB;
  const int64_t o_re = ((int64_t)kb * rows_total + rr) * SP_KB + quarter * 16;
  const int64_t o_im = o_re + SP_KB;
  const double sc = r < rows ? s[(int64_t)b * rows_pad + r] : 0.0;
  const double inv = sc > 0.0 ? 127.0 * (S == 4 ? 16777216.0 : 65536.0) / sc : 0.0;
  uint32_t wr[S][4], wi[S][4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t yr[4], yi[4], pr[S], pi[S];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = k0 + 4 * q + e;
      double2 v = make_double2(0.0, 0.0);
      if (r < rows && k < K) v = src.get(b, r, k);
      yr[e] = round_mul(v.x, inv);
      yi[e] = round_mul(v.y, inv);
    }
    digit_planes<S>(yr, pr);
    digit_planes<S>(yi, pi);
#pragma unroll
    for (int t = 0; t < S; ++t) wr[t][q] = pr[t], wi[t][q] = pi[t];
  }
#pragma unroll
  for (int t = 0; t < S; ++t) {
    *reinterpret_cast<uint4*>(planes + o_re + t * pstride) = make_uint4(wr[t][0], wr[t][1], wr[t][2], wr[t][3]);
    *reinterpret_cast<uint4*>(planes + o_im + t * pstride) = make_uint4(wi[t][0], wi[t][1], wi[t][2], wi[t][3]);
  }
}

// Bytes of scratch for one launch group of `nbatch` batches (planes and scales).
size_t sgemm_workspace_bytes(int nbatch, int M, int ncol, int K) {
  const int64_t mt = (M + SP_TILE - 1) / SP_TILE, nt = (ncol + SP_TILE - 1) / SP_TILE;
  const int64_t kp = (int64_t)align_up((size_t)std::min(std::max(K, 1), SP_SLAB), SP_KB);
  return align_up((size_t)SP_SA * kp * nbatch * mt * SP_ROWS, 1024) +
         align_up((size_t)SP_SB * kp * nbatch * nt * SP_ROWS, 1024) +
         align_up(sizeof(double) * nbatch * mt * SP_TILE, 256) +
         align_up(sizeof(double) * nbatch * nt * SP_TILE, 256) + 2048;
}

// The interstitial product GEMM on int8 slices for `nbatch` k points: A rows from
// cpw_unocc (plane waves in the order kperm), B rows gathered from the convolved grids at
// the offsets koff of the same order.
int sgemm_products(spx_ctx* ctx, int nbatch, int M, int ncol, int K, const double2* A,
                   int64_t lda, int64_t a_bstride, const int* kperm, const double2* grid,
                   int64_t g_bstride, int64_t g_nstride, const int64_t* coff, const int* koff,
                   int ncin, double2* out, int64_t sO2, int64_t sOn, int64_t sOc, double alpha,
                   void* ws, size_t ws_bytes, cudaStream_t s, int* launches, bool overwrite) {
  if (nbatch <= 0 || M <= 0 || ncol <= 0 || K <= 0) return SPX_OK;
  const int mt = (M + SP_TILE - 1) / SP_TILE, nt = (ncol + SP_TILE - 1) / SP_TILE;
  const int64_t RA = (int64_t)mt * SP_ROWS, RB = (int64_t)nt * SP_ROWS;
  if ((int64_t)nbatch * RB > 2147483647LL || (int64_t)nbatch * mt * nt > 2147483647LL)
    return set_error(ctx, SPX_EINVAL, "product GEMM too large for one launch group");
  uint8_t* base = (uint8_t*)align_up((size_t)ws, 1024);
  const size_t need = sgemm_workspace_bytes(nbatch, M, ncol, K);
  if (!ws || ws_bytes < need + 1024) return set_error(ctx, SPX_ENOMEM, "split product scratch too small");
  const size_t smem = sizeof(SgSmem) + 1024;
  cudaFuncSetAttribute(split_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int rc;
  // k is cut into exact int32 slabs of at most 32768; each slab adds into the output
  for (int kbeg = 0; kbeg < K; kbeg += SP_SLAB) {
    const int Ks = std::min(SP_SLAB, K - kbeg);
    const int nkb = (int)(align_up((size_t)Ks, SP_KB) / SP_KB);
    const int64_t kp = (int64_t)nkb * SP_KB;
    int8_t* PA = (int8_t*)base;
    int8_t* PB = (int8_t*)(base + align_up((size_t)SP_SA * kp * nbatch * RA, 1024));
    double* sA = (double*)((uint8_t*)PB + align_up((size_t)SP_SB * kp * nbatch * RB, 1024));
    double* sB = (double*)((uint8_t*)sA + align_up(sizeof(double) * nbatch * mt * SP_TILE, 256));
    const int rows_a = mt * SP_TILE, rows_b = nt * SP_TILE;  // padded rows (complex) per batch
    SgSrcRows sa{A, lda, a_bstride, kperm + kbeg};
    SgSrcGather sb{grid, g_bstride, g_nstride, coff, koff + kbeg, ncin};
    if (Ks <= SGP_K) {
      sgemm_prep_kernel<SP_SA><<<dim3(rows_a, nbatch), SGP_T, 0, s>>>(sa, M, rows_a, Ks, nkb, nbatch, RA, sA, PA);
      sgemm_prep_kernel<SP_SB><<<dim3(rows_b, nbatch), SGP_T, 0, s>>>(sb, ncol, rows_b, Ks, nkb, nbatch, RB, sB, PB);
      *launches += 2;
    } else {
      sgemm_rowmax_kernel<<<dim3(rows_a, nbatch), 256, 0, s>>>(sa, M, rows_a, Ks, sA);
      sgemm_rowmax_kernel<<<dim3(rows_b, nbatch), 256, 0, s>>>(sb, ncol, rows_b, Ks, sB);
      const int64_t ta = (int64_t)rows_a / 8 * 32 * nkb * nbatch, tb = (int64_t)rows_b / 8 * 32 * nkb * nbatch;
      sgemm_quant_kernel<SP_SA><<<(unsigned)((ta + 127) / 128), 128, 0, s>>>(sa, M, rows_a, Ks, nkb, nbatch, RA, sA, PA);
      sgemm_quant_kernel<SP_SB><<<(unsigned)((tb + 127) / 128), 128, 0, s>>>(sb, ncol, rows_b, Ks, nkb, nbatch, RB, sB, PB);
      *launches += 4;
    }
    if ((rc = check_cuda(ctx, cudaGetLastError(), "split product operand preparation"))) return rc;
    CUtensorMap mapA, mapB;
    const uint64_t rta = (uint64_t)nbatch * RA, rtb = (uint64_t)nbatch * RB;
    const uint64_t da[4] = {SP_KB, rta, (uint64_t)nkb, SP_SA};
    const uint64_t sta[3] = {SP_KB, rta * SP_KB, (uint64_t)nkb * rta * SP_KB};
    const uint32_t ba[4] = {SP_KB, SP_ROWS, 1, SP_SA};
    if ((rc = make_tmap_u8_4d(ctx, &mapA, PA, da, sta, ba, CU_TENSOR_MAP_SWIZZLE_64B))) return rc;
    const uint64_t db[4] = {SP_KB, rtb, (uint64_t)nkb, SP_SB};
    const uint64_t stb[3] = {SP_KB, rtb * SP_KB, (uint64_t)nkb * rtb * SP_KB};
    const uint32_t bb[4] = {SP_KB, SP_ROWS, 1, SP_SB};
    if ((rc = make_tmap_u8_4d(ctx, &mapB, PB, db, stb, bb, CU_TENSOR_MAP_SWIZZLE_64B))) return rc;
    SgParams prm;
    prm.nbatch = nbatch;
    prm.mtiles = mt;
    prm.ntiles = nt;
    prm.nitems = nbatch * mt * nt;
    prm.nk = nkb;
    prm.RA = RA;
    prm.RB = RB;
    prm.M = M;
    prm.ncol = ncol;
    prm.ncin = ncin;
    prm.sA = sA;
    prm.sB = sB;
    prm.out = reinterpret_cast<double*>(out);
    prm.sO2 = sO2;
    prm.sOn = sOn;
    prm.sOc = sOc;
    prm.alpha = alpha;
    prm.overwrite = overwrite && kbeg == 0;  // later K slabs add to the first
    prm.status = ctx->d_status;
    prm.timeout_ns = (uint64_t)(ctx->opt.timeout_ms > 0 ? ctx->opt.timeout_ms : 4000) * 1000000ull;
    const int grid_n = std::min(prm.nitems, ctx->num_sms);
    split_gemm_kernel<<<grid_n, SP1_THREADS, smem, s>>>(mapA, mapB, prm);
    if ((rc = check_cuda(ctx, cudaGetLastError(), "split_gemm_kernel launch"))) return rc;
    *launches += 1;
  }
  return SPX_OK;
}

}  // namespace spx
