// Dielectric matrix and its inverse in FP64 (src/correlation.f:614-636, :703-745).
//
// For every imaginary frequency the reference turns the packed polarisation into
//   eps_ij = delta_ij - sqrt(v_i) chi_ij sqrt(v_j)          (p_diagmatdiag, p_plusdiag)
// with v the Coulomb eigenvalues of the basis (the Coulomb-eigenbasis transform has
// made v diagonal), and inverts it as a packed Hermitian matrix (LAPACK zpptrf/zpptri
// on one process, ScaLAPACK with MPI). On the imaginary axis chi is negative
// semi-definite, so eps = 1 + (positive semi-definite) is positive definite. At
// Gamma the 3x3 head becomes 1 - 4 pi head and the wings -sqrt(4 pi) sqrt(v_i) wing.
//
// The inverse is computed here, for all frequencies at once, by the block sweep
// (Gauss-Jordan elimination without pivoting, which is stable for Hermitian positive
// definite matrices): for each 64-column pivot block k with P = inv(A_kk),
//   A_ij -= A_ik P A_kj,  A_ik <- A_ik P,  A_kj <- P A_kj,  A_kk <- -P   (i, j not in k),
// and after the last block A holds -inv(A). The pivot block is inverted by the same
// sweep one column at a time in shared memory; its pivots are the squares of the
// Cholesky pivots of A, so a pivot <= 0 marks a matrix that is not positive definite,
// reported with its frequency as zpptrf's info would be. The rank-64 updates run on
// the complex FP64 DMMA GEMM (K4c). The matrix stays Hermitian through the sweep, so
// only the 64 x 64 tiles on and above the diagonal are kept up to date: half of the
// multiply-adds and of the traffic of the updates. Measured at 24 matrices of 1200: 23.6 ms
// with full updates and the pivot block swept in shared memory, 8.4 ms here (updates
// 18.1 -> 6.3 ms: 0.72 of the FP64 pipe, a 64-deep tile's epilogue taking the rest; pivot
// blocks and panels 4.0 -> 0.86 ms).
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "spx_chain.cuh"
#include "spx_common.cuh"
#include "spx_zgemm.h"

namespace spx {

// full(i, j) = delta_ij - sq_i chi(i, j) sq_j for every frequency (grid.z), for the 64 x 64
// tiles on and above the diagonal; a CTA one column's 256 rows.
__global__ void dielec_unpack_kernel(const double2* __restrict__ chi, const double* __restrict__ sq,
                                     int n, double2* __restrict__ full) {
  const int j = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || (i >> 6) > (j >> 6)) return;
  const double2* c = chi + (int64_t)blockIdx.z * ((int64_t)n * (n + 1) / 2);
  double2 v;
  if (i <= j) {
    v = c[(int64_t)j * (j + 1) / 2 + i];
  } else {
    v = c[(int64_t)i * (i + 1) / 2 + j];
    v.y = -v.y;
  }
  const double s = -sq[i] * sq[j];
  double2 e = make_double2(s * v.x, s * v.y);
  if (i == j) e.x += 1.0;
  full[((int64_t)blockIdx.z * n + j) * n + i] = e;
}

__global__ void dielec_build_packed_kernel(double2* __restrict__ p, const double* __restrict__ sq,
                                           int n, int64_t npack, int nw) {
  const int64_t total = npack * nw;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ij = t % npack;
    int j = (int)((sqrt(8.0 * (double)ij + 1.0) - 1.0) * 0.5);
    while ((int64_t)j * (j + 1) / 2 > ij) --j;
    while ((int64_t)(j + 1) * (j + 2) / 2 <= ij) ++j;
    const int i = (int)(ij - (int64_t)j * (j + 1) / 2);
    const double s = -sq[i] * sq[j];
    double2 v = p[t];
    v.x *= s;
    v.y *= s;
    if (i == j) v.x += 1.0;
    p[t] = v;
  }
}

// packed(ij) = factor * full(i, j), i <= j, for every frequency (grid.y).
__global__ void pack_upper_kernel(const double2* __restrict__ full, int n, double factor,
                                  double2* __restrict__ packed) {
  const int64_t npack = (int64_t)n * (n + 1) / 2;
  const double2* fw = full + (int64_t)blockIdx.y * n * n;
  double2* pw = packed + (int64_t)blockIdx.y * npack;
  for (int64_t ij = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; ij < npack;
       ij += (int64_t)gridDim.x * blockDim.x) {
    int j = (int)((sqrt(8.0 * (double)ij + 1.0) - 1.0) * 0.5);
    while ((int64_t)j * (j + 1) / 2 > ij) --j;
    while ((int64_t)(j + 1) * (j + 2) / 2 <= ij) ++j;
    const int i = (int)(ij - (int64_t)j * (j + 1) / 2);
    const double2 v = fw[i + (int64_t)n * j];
    pw[ij] = make_double2(factor * v.x, factor * v.y);
  }
}

constexpr int DI_B = 64;  // pivot block of the sweep

// The panels of a pivot block move 16 rows x 64 columns t per CTA of 256 threads, four
// elements each; where rows and columns swap, through this tile, so that both sides move
// 256-byte runs.
using SweepTile = double2[4][16][17];

// After the trailing update, in the kept tiles: A(i, kb+t) = U(i, t) for rows i above the
// block, A(kb+t, j) = conj U(j, t) for columns j after it. Rows i0 .. i0 + 15 of U.
__device__ __forceinline__ void sweep_panels(SweepTile& tile, double2* Aw, int n, int kb, int bk, const double2* Uw,
                                             int i0) {
  const int lx = threadIdx.x & 15, ly = threadIdx.x >> 4, i = i0 + lx;
  // 16 divides kb, and bk unless the block is the last one
  if (i0 >= kb && i0 < kb + bk) return;
  double2 v[4];
#pragma unroll
  for (int h = 0; h < 4; ++h)
    if (i < n && 16 * h + ly < bk) v[h] = Uw[(int64_t)(16 * h + ly) * n + i];
  if (i0 < kb) {
#pragma unroll
    for (int h = 0; h < 4; ++h)
      if (16 * h + ly < bk) Aw[(int64_t)(kb + 16 * h + ly) * n + i] = v[h];
    return;
  }
#pragma unroll
  for (int h = 0; h < 4; ++h) tile[h][ly][lx] = v[h];
  __syncthreads();
  const int j = i0 + ly;
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const int t = 16 * h + lx;
    if (j < n && t < bk) Aw[(int64_t)j * n + kb + t] = make_double2(tile[h][lx][ly].x, -tile[h][lx][ly].y);
  }
}
__global__ void __launch_bounds__(256) sweep_panels_kernel(double2* A, int n, int kb, int bk, const double2* U) {
  __shared__ SweepTile tile;
  await_previous();
  const int64_t f = blockIdx.y;
  sweep_panels(tile, A + f * n * n, n, kb, bk, U + f * n * DI_B, 16 * blockIdx.x);
}

// CpT[j][t] = A(j, kb + t) for the rows j of one frequency outside the pivot block (its
// column panel, stored row by row; nothing reads the block's own rows of CpT or of U, and
// its tiles of A are being replaced). Rows below the pivot block come from its row panel,
// conjugated; rows of the pivot block before it, whose panels are not in A yet, from its U.
// Rows j0 .. j0 + 15.
__device__ __forceinline__ void sweep_extract(SweepTile& tile, const double2* Aw, int n, int kb, int bk,
                                              const double2* Uw, double2* __restrict__ Cw, int j0) {
  const int lx = threadIdx.x & 15, ly = threadIdx.x >> 4, j = j0 + ly;
  if (j0 >= kb && j0 < kb + bk) return;
  double2 v[4];
  if (j0 < kb - DI_B) {
#pragma unroll
    for (int h = 0; h < 4; ++h)
      if (16 * h + ly < bk) v[h] = Aw[(int64_t)(kb + 16 * h + ly) * n + j0 + lx];
#pragma unroll
    for (int h = 0; h < 4; ++h) tile[h][ly][lx] = v[h];
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 4; ++h)
      if (16 * h + lx < bk) Cw[(int64_t)j * DI_B + 16 * h + lx] = tile[h][lx][ly];
    return;
  }
  const double2* src = j < kb ? Uw + (int64_t)(j - (kb - DI_B)) * n : Aw + (int64_t)j * n;
#pragma unroll
  for (int h = 0; h < 4; ++h)
    if (j < n && 16 * h + lx < bk) v[h] = src[kb + 16 * h + lx];
#pragma unroll
  for (int h = 0; h < 4; ++h)
    if (j < n && 16 * h + lx < bk) Cw[(int64_t)j * DI_B + 16 * h + lx] = make_double2(v[h].x, -v[h].y);
}

// Pb <- inv(P) and A's pivot block <- -inv(P) for the bk x bk Hermitian positive-definite
// pivot block P of every frequency (the first `nw` CTAs, one each), by the sweep of its
// columns; meanwhile the other CTAs extract the column panels and put the panels of the
// pivot block before into A from its U: no two touch the same elements. Inverse,
// extraction and panels took 39 + 14 + 13 us one after the other at 24 matrices of 1200, 45
// together. A pivot that is not positive records (block row + 1) in info[frequency]. The
// chain of 64 pivots is serial, so a step is kept short: thread (r, c) of 16 x 16 holds rows
// r + 16 x, columns c + 16 y in registers, the pivot's row and column go through shared
// memory, two buffers and one barrier per step. (Updating and publishing the next pivot's
// row, column and reciprocal ahead of the rest of a step gained nothing.)
__global__ void __launch_bounds__(256) sweep_pivot_kernel(double2* A, int n, int kb, int bk, int nw,
                                                          const double2* U, double2* __restrict__ CpT,
                                                          double2* __restrict__ Pb, int* __restrict__ info) {
  __shared__ double2 col[2][DI_B], row[2][DI_B];
  release_next();
  if ((int)blockIdx.x >= nw) {
    __shared__ SweepTile tile;
    const int e = blockIdx.x - nw, nx = (n + 15) / 16, g = e / nx, x = 16 * (e - g * nx);
    const int64_t f = g < nw ? g : g - nw;
    double2* Af = A + f * n * n;
    const double2* Uf = U + f * n * DI_B;
    if (g < nw) sweep_extract(tile, Af, n, kb, bk, Uf, CpT + f * n * DI_B, x);
    else sweep_panels(tile, Af, n, kb - DI_B, DI_B, Uf, x);
    return;
  }
  double2* Aw = A + (int64_t)blockIdx.x * n * n + (int64_t)kb * n + kb;
  double2* Pw = Pb + (int64_t)blockIdx.x * DI_B * DI_B;
  const int r = threadIdx.x >> 4, c = threadIdx.x & 15;
  double2 m[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int i = r + 16 * x, j = c + 16 * y;
      m[x][y] = i < bk && j < bk ? Aw[(int64_t)j * n + i] : make_double2(i == j ? 1.0 : 0.0, 0.0);
    }
#pragma unroll
  for (int pq = 0; pq < 4; ++pq) {
    for (int pr = 0; pr < 16; ++pr) {
      const int p = 16 * pq + pr, b = p & 1;
      if (p >= bk) break;
      if (c == pr)
#pragma unroll
        for (int x = 0; x < 4; ++x) col[b][r + 16 * x] = m[x][pq];
      if (r == pr)
#pragma unroll
        for (int y = 0; y < 4; ++y) row[b][c + 16 * y] = m[pq][y];
      __syncthreads();
      const double piv = row[b][p].x;
      double d = 0.0;
      if (piv > 0.0) {
        d = 1.0 / piv;
      } else if (threadIdx.x == 0 && info[blockIdx.x] == 0) {
        info[blockIdx.x] = kb + p + 1;
      }
      double2 cx[4], ry[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const double2 u = col[b][r + 16 * x];
        cx[x] = make_double2(u.x * d, u.y * d);
      }
#pragma unroll
      for (int y = 0; y < 4; ++y) ry[y] = row[b][c + 16 * y];
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          const bool ip = x == pq && r == pr, jp = y == pq && c == pr;
          if (ip && jp) {
            m[x][y] = make_double2(-d, 0.0);
          } else if (jp) {
            m[x][y] = cx[x];
          } else if (ip) {
            m[x][y] = make_double2(ry[y].x * d, ry[y].y * d);
          } else {
            // m_ij - m_ip m_pj / m_pp
            m[x][y].x -= cx[x].x * ry[y].x - cx[x].y * ry[y].y;
            m[x][y].y -= cx[x].x * ry[y].y + cx[x].y * ry[y].x;
          }
        }
    }
  }
  // the sweep of every column leaves -inv
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const int i = r + 16 * x, j = c + 16 * y;
      if (i < bk && j < bk) {
        Pw[i * DI_B + j] = make_double2(-m[x][y].x, -m[x][y].y);
        Aw[(int64_t)j * n + i] = m[x][y];
      }
    }
}

// head(:, f) = I3 - 4 pi head(:, f) (packed 3x3), wing(:, i, f) = -sqrt(4 pi) sqrt(v_i) wing
__global__ void dielec_headwing_kernel(double2* head, double2* wing, const double* __restrict__ sq,
                                       int n, int nw) {
  const double fourpi = 4.0 * 3.14159265358979323846;
  const double sfp = sqrt(fourpi);
  const int64_t nh = 6LL * nw, ng = wing ? 3LL * n * nw : 0;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nh + ng;
       t += (int64_t)gridDim.x * blockDim.x) {
    if (t < nh) {
      if (!head) continue;
      const int ij = (int)(t % 6);
      double2 v = head[t];
      v.x = -fourpi * v.x;
      v.y = -fourpi * v.y;
      if (ij == 0 || ij == 2 || ij == 5) v.x += 1.0;
      head[t] = v;
    } else {
      const int64_t u = t - nh;
      const int i = (int)((u / 3) % n);
      const double f = -sfp * sq[i];
      double2 v = wing[u];
      wing[u] = make_double2(f * v.x, f * v.y);
    }
  }
}

__global__ void sqrt_kernel(const double* __restrict__ v, double* __restrict__ s, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    s[i] = sqrt(v[i]);
}

void dielec_release(spx_ctx* ctx) { ctx->dn = nullptr; }

}  // namespace spx

using namespace spx;

extern "C" int spx_dielec_dev(spx_ctx* ctx, int32_t nbas, int32_t nw, double* susceph,
                              const double* coul, int32_t invert, double* head, double* wing,
                              void* stream) {
  if (!ctx) return SPX_EINVAL;
  if (nbas < 0 || nw < 0) return set_error(ctx, SPX_EINVAL, "negative size");
  if (nbas == 0 || nw == 0) return SPX_OK;
  if (!susceph || !coul) return set_error(ctx, SPX_EINVAL, "null array argument");
  if (nbas > 46340) return set_error(ctx, SPX_EINVAL, "nbas too large for packed indexing");
  cudaSetDevice(ctx->device);
  cudaStream_t s = pick_stream(ctx, stream);
  const int n = nbas;
  const int64_t npack = (int64_t)n * (n + 1) / 2;
  const int grid = ctx->num_sms * 8;
  int rc;
  // scratch: sqrt(v), infos, and for the inversion the full matrices of every
  // frequency, the pivot blocks, the column panels and their products
  size_t need = align_up(sizeof(double) * n, 256) + align_up(sizeof(int) * nw, 256);
  const size_t full_b = align_up(sizeof(double2) * (size_t)n * n * nw, 256);
  const size_t pan_b = align_up(sizeof(double2) * (size_t)n * DI_B * nw, 256);
  const size_t blk_b = align_up(sizeof(double2) * (size_t)DI_B * DI_B * nw, 256);
  if (invert) need += full_b + 2 * pan_b + blk_b;
  if ((rc = ensure_workspace(ctx, need + 1024))) return rc;
  char* b = (char*)ctx->ws;
  double* sq = (double*)b;
  b += align_up(sizeof(double) * n, 256);
  int* info = (int*)b;
  b += align_up(sizeof(int) * nw, 256);
  sqrt_kernel<<<(n + 255) / 256, 256, 0, s>>>(coul, sq, n);
  if ((rc = check_cuda(ctx, cudaGetLastError(), "sqrt_kernel launch"))) return rc;
  double2* P = reinterpret_cast<double2*>(susceph);
  if (head || wing) {
    dielec_headwing_kernel<<<grid, 256, 0, s>>>(reinterpret_cast<double2*>(head),
                                                reinterpret_cast<double2*>(wing), sq, n, nw);
    if ((rc = check_cuda(ctx, cudaGetLastError(), "dielec_headwing_kernel launch"))) return rc;
  }
  if (!invert) {
    dielec_build_packed_kernel<<<grid, 256, 0, s>>>(P, sq, n, npack, nw);
    return check_cuda(ctx, cudaGetLastError(), "dielec_build_packed_kernel launch");
  }
  double2* full = reinterpret_cast<double2*>(b);
  b += full_b;
  double2* CpT = reinterpret_cast<double2*>(b);
  b += pan_b;
  double2* U = reinterpret_cast<double2*>(b);
  b += pan_b;
  double2* Pb = reinterpret_cast<double2*>(b);
  if ((rc = check_cuda(ctx, cudaMemsetAsync(info, 0, sizeof(int) * nw, s), "zero info"))) return rc;
  for (int f = 0; f < nw; f += 65535) {   // grid.z limit
    const int nf = std::min(nw - f, 65535);
    dielec_unpack_kernel<<<dim3((n + 255) / 256, n, nf), 256, 0, s>>>(P + (int64_t)f * npack, sq, n,
                                                                      full + (int64_t)f * n * n);
    if ((rc = check_cuda(ctx, cudaGetLastError(), "dielec_unpack_kernel launch"))) return rc;
  }
  const int nx = (n + 15) / 16;
  for (int kb = 0; kb < n; kb += DI_B) {
    const int bk = std::min(DI_B, n - kb);
    // the GEMMs follow this kernel as a chain; not it them: its first CTAs, the serial
    // inverses, would land in pairs on the SMs that drain first (24 of 1200: 8.4 -> 8.7 ms)
    sweep_pivot_kernel<<<nw * (1 + nx * (kb ? 2 : 1)), 256, 0, s>>>(full, n, kb, bk, nw, U, CpT, Pb, info);
    if ((rc = check_cuda(ctx, cudaGetLastError(), "sweep pivot block"))) return rc;
    // U = Cp P: U(i, c) = sum_t Cp(i, t) conj(P(c, t))   (P Hermitian)
    ZgParams g{};
    g.A = CpT;
    g.lda = DI_B;
    g.sA1 = (int64_t)n * DI_B;
    g.B = Pb;
    g.sB1 = (int64_t)DI_B * DI_B;
    g.sBc = DI_B;
    g.O = U;
    g.sO1 = (int64_t)n * DI_B;
    g.sOc = n;
    g.alpha_v = make_double2(1.0, 0.0);
    g.M = n;
    g.ncol = bk;
    g.ncin = bk;
    g.K = bk;
    g.nb1 = nw;
    g.overwrite = 1;
    if ((rc = launch_zgemm(ctx, g, nw, s, true))) return rc;
    // A(i, j) -= sum_t U(i, t) conj(Cp(j, t))   (= U_i A_kj, A Hermitian)
    ZgParams h{};
    h.A = U;
    h.a_mcontig = 1;
    h.lda = n;
    h.sA1 = (int64_t)n * DI_B;
    h.B = CpT;
    h.sB1 = (int64_t)n * DI_B;
    h.sBc = DI_B;
    h.O = full;
    h.sO1 = (int64_t)n * n;
    h.sOc = n;
    h.alpha_v = make_double2(-1.0, 0.0);
    h.M = n;
    h.ncol = n;
    h.ncin = n;
    h.K = bk;
    h.nb1 = nw;
    h.upper = 1;
    h.skip = kb / DI_B + 1;   // the panels replace these tiles: 171 of 190 are left at n = 1200
    if ((rc = launch_zgemm(ctx, h, nw, s, true))) return rc;
    if (kb + bk < n) continue;
    if ((rc = check_cuda(ctx, launch_chained(sweep_panels_kernel, dim3(nx, nw), 256, 0, s, true, full, n, kb, bk, U),
                         "sweep panels")))
      return rc;
  }
  // the sweep leaves -inv(eps)
  pack_upper_kernel<<<dim3(grid, nw), 256, 0, s>>>(full, n, -1.0, P);
  if ((rc = check_cuda(ctx, cudaGetLastError(), "pack_upper_kernel launch"))) return rc;
  std::vector<int> hinfo(nw);
  if ((rc = check_cuda(ctx, cudaMemcpyAsync(hinfo.data(), info, sizeof(int) * nw, cudaMemcpyDeviceToHost, s),
                       "copy info")) ||
      (rc = check_cuda(ctx, cudaStreamSynchronize(s), "dielectric inversion")))
    return rc;
  for (int f = 0; f < nw; ++f)
    if (hinfo[f] != 0)
      return set_error(ctx, SPX_EINVAL,
                       "dielectric matrix of frequency " + std::to_string(f) +
                           " is not positive definite (pivot " + std::to_string(hinfo[f]) + ")");
  return SPX_OK;
}
