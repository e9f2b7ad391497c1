// K5: the FFT branch of the interstitial products (src/wavefproducts.f:576-758).
//
// The reference, per k point: scatters each band's plane-wave coefficients to an
// nfft^3 grid and transforms G -> r (FFTW_BACKWARD); the occupied bands become
// conj(phi_n(r))/sqrt(vol) times the step function theta(r), the unoccupied
// ones phi_n'(r)/nnfft; every pair's pointwise product is transformed r -> G
// (FFTW_FORWARD) and the mixed-basis plane waves G_M - g are gathered out of it.
//
// Here only what the gather needs is computed. Grids are [band][z][y][x], x contiguous:
//   * band grids (K5a, `dft_line_kernel`, `dft_across_kernel` x2): the coefficients live in
//     a small G box, so each of the three separable passes sums only over the box
//     extent of its axis (19 of 48 for a 3000-wave sphere on a 48^3 grid); the last pass applies
//     conj, 1/sqrt(vol), theta or 1/nnfft;
//   * pair x and y passes (K5b) at fixed z, keeping the kx and ky values that occur in
//     G_M - g only (13 of 48 each), then the z pass and gather (K5c) for exactly the
//     (kx, ky, kz) of each G_M, added into cprod's column.
// Mixed-basis vectors that reach at most 7 from the origin on each axis (`sym`), which is
// every sphere of up to 1400 of them, take the folded passes on the FP64 tensor cores
// (`fft_pair_fold_kernel`, `fft_pair_gather_kernel`); the backfolding vector g goes into
// the step function's transform there. Other sets sum the pruned transforms on the CUDA
// cores: grid edges n = 16 r (r <= 4) with a radix-16 x r line FFT
// (`fft_pair_zy_radix_kernel`), other edges directly (`fft_pair_zy_kernel`); their "z" is
// the line axis x here, and `fft_pair_x_kernel` runs over z.
// All arithmetic is FP64; the twiddles are tables of cos and sin of 2 pi m / nfft.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "spx_common.cuh"
#include "spx_dmma.cuh"

namespace spx {

constexpr int FFT_NMAX = 64;   // largest grid edge
constexpr int FFT_KMAX = 16;   // largest number of distinct G_M - g values per axis
constexpr int FFT_NP = 4;      // unoccupied bands per K5b CTA
constexpr int FFT_XC = 8;      // x planes staged per K5c step

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ void cfma(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}

// The separable DFT passes of the band grids, G (box index i, value lo + i) -> r (j):
//   out(j) = sum_i in(i) exp(+2 pi i (lo + i) j / n).
// With Pc = sum in cos and Ps = sum in sin, out(j) = Pc + i Ps and out(n - j) = Pc - i Ps: a
// thread owns such pairs of outputs, which halves the multiply-adds, the loads and the
// table reads per output.

// First pass, along contiguous lines: in (nline, nin) -> out (nline, n); a thread one output
// pair of one line.
__global__ void __launch_bounds__(256)
    dft_line_kernel(const double2* __restrict__ in, double2* __restrict__ out,
                    const double2* __restrict__ twb, int nin, int lo, int n, int64_t nline) {
  __shared__ double2 tw[FFT_NMAX];
  for (int i = threadIdx.x; i < n; i += blockDim.x) tw[i] = twb[i];
  __syncthreads();
  const int nh = n / 2 + 1;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nline * nh;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t line = t / nh;
    const int j = (int)(t - line * nh);
    const double2* src = in + line * nin;
    int m = ((lo * j) % n + n) % n;
    double2 pc = make_double2(0.0, 0.0), ps = pc;
    for (int i = 0; i < nin; ++i) {
      const double2 v = __ldg(src + i), w = tw[m];
      pc.x = fma(v.x, w.x, pc.x);
      pc.y = fma(v.y, w.x, pc.y);
      ps.x = fma(v.x, w.y, ps.x);
      ps.y = fma(v.y, w.y, ps.y);
      m += j;
      if (m >= n) m -= n;
    }
    double2* o = out + line * n;
    o[j] = make_double2(pc.x - ps.y, pc.y + ps.x);
    if (j > 0 && n - j > j) o[n - j] = make_double2(pc.x + ps.y, pc.y - ps.x);
  }
}

// Second and third pass, across lines: for every outer (o1, o2) and x < n (contiguous on both
// sides), in[o1 i1 + o2 i2 + i is + x] -> out[o1 s1 + o2 s2 + j sj + x], then optionally
// conj, times scale, times mul[o2 m2 + j mj + x]. A thread owns one x and DFT_JP output
// pairs, so an input serves 2 DFT_JP outputs; the table reads are the same for a whole warp's
// group of pairs. Bound by their latency, so three CTAs per SM (80 registers, a few spilled)
// beat two: 600 bands of 19^3 to 48^3, z pass 0.59 against 0.73 ms (1.81 ms with one output per
// thread).
constexpr int DFT_JP = 5;
struct DftAcross {
  const double2* in;
  double2* out;
  const double2* tw;   // exp(+2 pi i m / n), m < n
  const double2* mul;  // or null
  int nin, lo, n, n2;  // o2 < n2
  int64_t outer;       // o1 n2 + o2
  int64_t is, i1, i2, sj, s1, s2, mj, m2;
  double scale;
  int conj_out;
};

__global__ void __launch_bounds__(256, 3) dft_across_kernel(DftAcross p) {
  __shared__ double2 tw[FFT_NMAX];
  for (int i = threadIdx.x; i < p.n; i += blockDim.x) tw[i] = p.tw[i];
  __syncthreads();
  const int nh = p.n / 2 + 1, ng = (nh + DFT_JP - 1) / DFT_JP;
  // pairs past the last one repeat it and are not stored: a step of the table index
  // stays below n, so one subtraction keeps it in the table
  const int last = nh - 1;
  const int64_t total = p.outer * ng * p.n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = t / p.n;
    const int x = (int)(t - r * p.n);
    const int64_t o = r / ng;
    const int j0 = (int)(r - o * ng) * DFT_JP;
    const int64_t o1 = o / p.n2;
    const int o2 = (int)(o - o1 * p.n2);
    const double2* src = p.in + o1 * p.i1 + o2 * p.i2 + x;
    double2 pc[DFT_JP], ps[DFT_JP];
    int m[DFT_JP];
#pragma unroll
    for (int k = 0; k < DFT_JP; ++k) {
      pc[k] = ps[k] = make_double2(0.0, 0.0);
      m[k] = ((p.lo * min(j0 + k, last)) % p.n + p.n) % p.n;
    }
#pragma unroll 2
    for (int i = 0; i < p.nin; ++i) {
      const double2 v = __ldg(src + i * p.is);
#pragma unroll
      for (int k = 0; k < DFT_JP; ++k) {
        const double2 w = tw[m[k]];
        pc[k].x = fma(v.x, w.x, pc[k].x);
        pc[k].y = fma(v.y, w.x, pc[k].y);
        ps[k].x = fma(v.x, w.y, ps[k].x);
        ps[k].y = fma(v.y, w.y, ps[k].y);
        m[k] += min(j0 + k, last);
        if (m[k] >= p.n) m[k] -= p.n;
      }
    }
    double2* dst = p.out + o1 * p.s1 + o2 * p.s2 + x;
    const double2* mul = p.mul ? p.mul + o2 * p.m2 + x : nullptr;
    auto put = [&](int j, double2 v) {
      if (p.conj_out) v.y = -v.y;
      v.x *= p.scale;
      v.y *= p.scale;
      if (mul) v = cmul(v, mul[j * p.mj]);
      dst[j * p.sj] = v;
    };
#pragma unroll
    for (int k = 0; k < DFT_JP; ++k) {
      const int j = j0 + k;
      if (j >= nh) continue;
      put(j, make_double2(pc[k].x - ps[k].y, pc[k].y + ps[k].x));
      if (j > 0 && p.n - j > j) put(p.n - j, make_double2(pc[k].x + ps[k].y, pc[k].y - ps[k].x));
    }
  }
}

// box[b*size + gidx[i]] = cpw[b*ngpt + i]; the box is zeroed beforehand.
__global__ void fft_scatter_kernel(const double2* __restrict__ cpw, int ngpt,
                                   const int* __restrict__ gidx, int64_t size,
                                   double2* __restrict__ box) {
  const int64_t b = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ngpt; i += gridDim.x * blockDim.x)
    box[b * size + gidx[i]] = cpw[b * ngpt + i];
}

struct PairParams {
  const double2* A;    // [kl*nocc + n][x][y][z]
  const double2* B;    // [kl*nunocc + n'][x][y][z]
  double2* T2;         // [pairc][x][kz][ky]
  const double2* twf;  // exp(-2 pi i m / n)
  const int* kz;       // distinct kz values (nkz)
  const int* ky;
  int n, nocc, nunocc, nkz, nky;
};

// grid (kl*nocc + n, unoccupied group, x); block (n threads along y, FFT_NP bands)
__global__ void __launch_bounds__(FFT_NMAX * FFT_NP) fft_pair_zy_kernel(PairParams p) {
  extern __shared__ double2 sm[];
  const int n = p.n;
  double2* Apl = sm;                               // [y][z]
  double2* Ez = Apl + n * n;                       // [kk][z]
  double2* Ey = Ez + FFT_KMAX * n;                 // [kk][y]
  double2* T1 = Ey + FFT_KMAX * n;                 // [j][kz][y]
  const int kn = blockIdx.x, grp = blockIdx.y, x = blockIdx.z;
  const int kl = kn / p.nocc;
  const int tid = threadIdx.y * blockDim.x + threadIdx.x, nth = blockDim.x * blockDim.y;
  const double2* a = p.A + ((int64_t)kn * n + x) * n * n;
  for (int i = tid; i < n * n; i += nth) Apl[i] = a[i];
  for (int i = tid; i < FFT_KMAX * n; i += nth) {
    const int kk = i / n, z = i - kk * n;
    Ez[i] = kk < p.nkz ? p.twf[(p.kz[kk] * z) % n] : make_double2(0.0, 0.0);
    Ey[i] = kk < p.nky ? p.twf[(p.ky[kk] * z) % n] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const int y = threadIdx.x, j = threadIdx.y;
  const int np = grp * FFT_NP + j;
  if (np < p.nunocc) {
    const double2* bl = p.B + (((int64_t)kl * p.nunocc + np) * n + x) * n * n + (int64_t)y * n;
    const double2* al = Apl + y * n;
    double2 acc[FFT_KMAX];
#pragma unroll
    for (int kk = 0; kk < FFT_KMAX; ++kk) acc[kk] = make_double2(0.0, 0.0);
    for (int z = 0; z < n; ++z) {
      const double2 prod = cmul(al[z], __ldg(bl + z));
#pragma unroll
      for (int kk = 0; kk < FFT_KMAX; ++kk)
        if (kk < p.nkz) cfma(acc[kk], Ez[kk * n + z], prod);
    }
    for (int kk = 0; kk < p.nkz; ++kk) T1[(j * FFT_KMAX + kk) * n + y] = acc[kk];
  }
  __syncthreads();
  // y pass: T2[pair][x][kz][ky] = sum_y Ey[ky][y] T1[j][kz][y]
  const int nout = FFT_NP * p.nkz * p.nky;
  for (int o = tid; o < nout; o += nth) {
    const int jj = o / (p.nkz * p.nky);
    const int rem = o - jj * p.nkz * p.nky;
    const int kz = rem / p.nky, ky = rem - kz * p.nky;
    const int npp = grp * FFT_NP + jj;
    if (npp >= p.nunocc) continue;
    const double2* t1 = T1 + (jj * FFT_KMAX + kz) * n;
    const double2* ey = Ey + ky * n;
    double2 s = make_double2(0.0, 0.0);
    for (int yy = 0; yy < n; ++yy) cfma(s, ey[yy], t1[yy]);
    const int64_t pairc = (int64_t)kn * p.nunocc + npp;
    p.T2[((pairc * n + x) * p.nkz + kz) * p.nky + ky] = s;
  }
}

// ---------------------------------------------------------------------------
// K5b as a line FFT, for grid edges n = 16 r (r = 1..4): the 48-point transform of
// the 48^3 grid is radix 16 x 3. With z = r n1 + n2 and k = k1 + 16 k2,
//   X[k] = sum_{n2<r} W_n^{n2 k1} W_r^{n2 k2} F_{n2}[k1],
//   F_{n2}[k1] = sum_{n1<16} x[r n1 + n2] W_16^{n1 k1},
// so thread (line, n2) transforms its 16 decimated points in registers (radix 4 x 4),
// applies W_n^{n2 k1}, and the r partial spectra of a line are combined, through
// shared memory, only at the k the gather needs. W = exp(-2 pi i / n) (forward).

// 4-point forward DFT in place: (x0, x1, x2, x3) -> (X0, X1, X2, X3), W_4 = -i.
__device__ __forceinline__ void dft4_fwd(double2& x0, double2& x1, double2& x2, double2& x3) {
  const double2 t0 = make_double2(x0.x + x2.x, x0.y + x2.y), t1 = make_double2(x0.x - x2.x, x0.y - x2.y);
  const double2 t2 = make_double2(x1.x + x3.x, x1.y + x3.y), t3 = make_double2(x1.x - x3.x, x1.y - x3.y);
  x0 = make_double2(t0.x + t2.x, t0.y + t2.y);
  x2 = make_double2(t0.x - t2.x, t0.y - t2.y);
  x1 = make_double2(t1.x + t3.y, t1.y - t3.x);  // t1 - i t3
  x3 = make_double2(t1.x - t3.y, t1.y + t3.x);  // t1 + i t3
}

// 16-point forward DFT of v (natural order in): n1 = 4a + b, k1 = c + 4d; 4-point
// transforms over a, twiddles W_16^{bc} (w16[m] = W_16^m), 4-point transforms over b.
// The output is left digit-reversed: X[k1] is v[fft16_pos(k1)].
__host__ __device__ constexpr int fft16_pos(int k1) { return 4 * (k1 & 3) + (k1 >> 2); }
__device__ __forceinline__ void fft16_fwd(double2 (&v)[16], const double2* __restrict__ w16) {
#pragma unroll
  for (int b = 0; b < 4; ++b) dft4_fwd(v[b], v[4 + b], v[8 + b], v[12 + b]);  // v[4c + b] = Y_b[c]
#pragma unroll
  for (int b = 1; b < 4; ++b)
#pragma unroll
    for (int c = 1; c < 4; ++c) v[4 * c + b] = cmul(v[4 * c + b], w16[b * c]);
#pragma unroll
  for (int c = 0; c < 4; ++c) dft4_fwd(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);  // v[4c + d] = X[c + 4d]
}

// Shared-memory row strides of the line FFT: 17 complex per (line, phase) spectrum and
// n + 1 per kz row, so that lanes walking lines hit distinct banks.
constexpr int FFTR_LD = 17;

struct PairFftParams {
  const double2* A;    // [kl*nocc + n][x][y][z]
  const double2* B;    // [kl*nunocc + n'][x][y][z]
  double2* T2;         // [pairc][x][kz][ky]
  const double2* twf;  // W_n^m = exp(-2 pi i m / n), m < n
  const int* kz;       // distinct kz values (nkz)
  const int* ky;
  int n, r, bpc, nocc, nunocc, nkz, nky;
};

// grid (kl*nocc + n, group of bpc unoccupied bands, x); block bpc * n * r threads:
// thread t of band j is line t / r, decimation phase t % r.
__global__ void __launch_bounds__(512) fft_pair_zy_radix_kernel(PairFftParams p) {
  extern __shared__ double2 smr[];
  const int n = p.n, r = p.r, per = n * r;
  double2* tw = smr;                                 // [n]
  double2* w16 = tw + n;                             // [16]
  double2* Fb = w16 + 16;                            // [bpc][n lines][r][FFTR_LD]
  double2* T1 = Fb + (size_t)p.bpc * n * r * FFTR_LD;  // [bpc][FFT_KMAX][n + 1]
  const int kn = blockIdx.x, grp = blockIdx.y, x = blockIdx.z;
  const int kl = kn / p.nocc;
  for (int i = threadIdx.x; i < n; i += blockDim.x) tw[i] = p.twf[i];
  for (int i = threadIdx.x; i < 16; i += blockDim.x) w16[i] = p.twf[i * r];
  __syncthreads();
  const int j = threadIdx.x / per, t = threadIdx.x - j * per;
  const int np = grp * p.bpc + j;
  const bool live = j < p.bpc && np < p.nunocc;
  double2* F = Fb + (size_t)j * n * r * FFTR_LD;
  double2* T = T1 + (size_t)j * FFT_KMAX * (n + 1);
  const int tl = n + 1;
  // z pass: line y = t / r of the product plane A(x, y, .) B(x, y, .)
  if (live) {
    const int y = t / r, n2 = t - (t / r) * r;
    const double2* a = p.A + (((int64_t)kn * n + x) * n + y) * n;
    const double2* bl = p.B + ((((int64_t)kl * p.nunocc + np) * n + x) * n + y) * n;
    double2 v[16];
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) {
      const int z = r * n1 + n2;
      v[n1] = cmul(__ldg(a + z), __ldg(bl + z));
    }
    fft16_fwd(v, w16);
    double2* f = F + ((size_t)y * r + n2) * FFTR_LD;
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1) f[k1] = n2 ? cmul(v[fft16_pos(k1)], tw[n2 * k1]) : v[fft16_pos(k1)];
  }
  __syncthreads();
  // combine at the needed kz: T[kk][y]
  if (live) {
    for (int o = t; o < p.nkz * n; o += per) {
      const int kk = o / n, y = o - kk * n;
      const int k = p.kz[kk], k1 = k & 15, k2 = k >> 4;
      const double2* f = F + (size_t)y * r * FFTR_LD + k1;
      double2 acc = f[0];
      for (int n2 = 1; n2 < r; ++n2) cfma(acc, f[n2 * FFTR_LD], tw[(16 * n2 * k2) % n]);
      T[kk * tl + y] = acc;
    }
  }
  __syncthreads();
  // y pass: line kk of T along y
  if (live && t < p.nkz * r) {
    const int kk = t / r, n2 = t - (t / r) * r;
    double2 v[16];
#pragma unroll
    for (int n1 = 0; n1 < 16; ++n1) v[n1] = T[kk * tl + r * n1 + n2];
    fft16_fwd(v, w16);
    double2* f = F + ((size_t)kk * r + n2) * FFTR_LD;
#pragma unroll
    for (int k1 = 0; k1 < 16; ++k1) f[k1] = n2 ? cmul(v[fft16_pos(k1)], tw[n2 * k1]) : v[fft16_pos(k1)];
  }
  __syncthreads();
  if (live) {
    const int64_t pairc = (int64_t)kn * p.nunocc + np;
    double2* out = p.T2 + (pairc * n + x) * p.nkz * p.nky;
    for (int o = t; o < p.nkz * p.nky; o += per) {
      const int kk = o / p.nky, kyi = o - kk * p.nky;
      const int k = p.ky[kyi], k1 = k & 15, k2 = k >> 4;
      const double2* f = F + (size_t)kk * r * FFTR_LD + k1;
      double2 acc = f[0];
      for (int n2 = 1; n2 < r; ++n2) cfma(acc, f[n2 * FFTR_LD], tw[(16 * n2 * k2) % n]);
      out[o] = acc;
    }
  }
}

struct GatherParams {
  const double2* T2;   // [pairc][x][kz][ky]
  const double2* twf;
  const int* kx;       // distinct kx values
  const int* gmap;     // per ig: ix | iy << 8 | iz << 16
  double2* cprod;      // already offset to (first pair of the chunk, column col0)
  int64_t ldc;
  int n, nkx, nky, nkz, ngptm;
};

// grid: one CTA per pair of the chunk
__global__ void __launch_bounds__(256) fft_pair_x_kernel(GatherParams p) {
  extern __shared__ double2 sm[];
  const int n = p.n, plane = p.nkz * p.nky;
  double2* Ex = sm;                        // [kk][x]
  double2* F = Ex + FFT_KMAX * n;          // [ig]
  double2* Ts = F + p.ngptm;               // [xc][kz][ky]
  const int64_t pairc = blockIdx.x;
  for (int i = threadIdx.x; i < FFT_KMAX * n; i += blockDim.x) {
    const int kk = i / n, x = i - kk * n;
    Ex[i] = kk < p.nkx ? p.twf[(p.kx[kk] * x) % n] : make_double2(0.0, 0.0);
  }
  for (int i = threadIdx.x; i < p.ngptm; i += blockDim.x) F[i] = make_double2(0.0, 0.0);
  const double2* t2 = p.T2 + pairc * n * plane;
  for (int x0 = 0; x0 < n; x0 += FFT_XC) {
    const int xc = min(FFT_XC, n - x0);
    __syncthreads();
    for (int i = threadIdx.x; i < xc * plane; i += blockDim.x) Ts[i] = t2[(int64_t)x0 * plane + i];
    __syncthreads();
    for (int ig = threadIdx.x; ig < p.ngptm; ig += blockDim.x) {
      const int g = p.gmap[ig];
      const int ix = g & 255, iy = (g >> 8) & 255, iz = (g >> 16) & 255;
      double2 acc = F[ig];
      for (int xx = 0; xx < xc; ++xx) cfma(acc, Ex[ix * n + x0 + xx], Ts[xx * plane + iz * p.nky + iy]);
      F[ig] = acc;
    }
  }
  for (int ig = threadIdx.x; ig < p.ngptm; ig += blockDim.x) {
    double2* o = p.cprod + pairc + p.ldc * ig;
    double2 v = *o;
    v.x += F[ig].x;
    v.y += F[ig].y;
    *o = v;
  }
}

// ---------------------------------------------------------------------------
// K5b / K5c on the FP64 tensor cores, for k = 0 .. 7 and -7 .. -1 on each axis.
//
// A forward transform kept at +-k folds: with c_z = p_z + p_{n-z} and s_z = p_z - p_{n-z}
// (0 < z < n / 2; c_0 = p_0),
//   C_k = sum_z c_z cos(2 pi z k / n) (+ (-1)^k p_{n/2} for even n),  S_k = sum_z s_z sin(2 pi z k / n),
//   X_{+-k} = C_k -+ i S_k:
// real matrices of at most 8 x 32 (FFS_K = 8 frequencies) contract the real and imaginary parts
// separately, a quarter of the multiply-adds of a complex transform over all n, on
// FP64 mma.sync. A thread forms the folded products its fragment needs in registers.
//
// K5b: a warp owns one pair at one z plane. Lines come in
// chunks of 8 y slots: rows 0 .. 7 the lines y, rows 15 .. 8 their mirrors n - y (for y = 0 the line
// n / 2). m8n8k4 takes the frequencies as rows, slots as k and 8 lines as columns, so the
// x pass leaves (kx = g; lines 2t, 2t + 1) in a thread, and the same for the mirrors: folded
// there, they are the B fragments of the y pass (k = slots 2t, then 2t + 1; columns kx) as
// they stand, and nothing is exchanged. (All FP64 mma shapes run at the same rate, measured
// 36-37 TFLOP/s.) The y pass's 16 accumulators per pair live through the plane. The lines of
// NA + NB bands are copied by bulk copies, two chunks deep, by warp 0; NA NB pairs share
// them. Planes of one z run together, so the grids come from memory once. Bound: the FP64
// pipe (products, folds and mma share it); shared-memory reads take about half of its time.
// Measured on the 48^3 grid, 24000 pairs of 3000-wave bands, 13 values per axis: the pair
// passes 31.1 ms with the line FFT, 7.3 ms here (0.6 of the FP64 pipe; two pairs per warp and
// 8 warps 8.1 ms); the whole call 38.4 -> 9.5 ms.
constexpr int FFS_K = 8;
constexpr int FFS_ROWS = 16, FFS_SLOTS = 8;
constexpr int FFS_THREADS = 512;            // 16 warps of 128 registers

struct FoldParams {
  const double2* A;    // [kl nocc + n][z][y][ld]
  const double2* B;    // [kl nunocc + n'][z][y][ld]
  double2* T2;         // [pair][z][kx][ky]
  const double2* tab;  // [k][sl]: (cos, sin)(2 pi slot k / n), 0 for slots >= H
  const int* posx;     // index of k in the list of kx values, at k + 7 (-1: not needed)
  const int* posy;
  int n, ld, H, nst, sl;   // H = ceil(n / 2) slots, nst = ceil(H / 8), sl = 8 nst + 4
  int nk, nocc, nunocc, na, nb, nkx, nky;
  int ga, gb;              // groups of occupied / unoccupied bands
  int* status;
  uint64_t timeout_ns;
};

// X_{+-k} of (C, S) pairs: C - i S and C + i S.
__device__ __forceinline__ double2 fold_plus(double2 c, double2 s) { return make_double2(c.x + s.y, c.y - s.x); }
__device__ __forceinline__ double2 fold_minus(double2 c, double2 s) { return make_double2(c.x - s.y, c.y + s.x); }

__global__ void __launch_bounds__(FFS_THREADS, 1) fft_pair_fold_kernel(FoldParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nw = p.na * p.nb, nband = p.na + p.nb;
  const int bandsz = FFS_ROWS * p.ld;                         // double2 per band and stage
  double2* stage = reinterpret_cast<double2*>(smem_raw);      // [2][nband][16][ld]
  double2* tab = stage + 2 * (size_t)nband * bandsz;          // [8][sl]
  uint64_t* full = reinterpret_cast<uint64_t*>(tab + FFS_K * p.sl);
  uint64_t* empty = full + 2;
  int* pos = reinterpret_cast<int*>(empty + 2);               // [2][16]
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], nw);
    }
    fence_barrier_init();
  }
  for (int i = threadIdx.x; i < FFS_K * p.sl; i += blockDim.x) tab[i] = p.tab[i];
  if (threadIdx.x < 15) {
    pos[threadIdx.x] = p.posx[threadIdx.x];
    pos[16 + threadIdx.x] = p.posy[threadIdx.x];
  }
  __syncthreads();
  const int64_t per_z = (int64_t)p.nk * p.ga * p.gb, ntask = per_z * p.n;

  // warp 0 copies chunk `issued` of this CTA's sequence: lane b the lines of band b, into the
  // stage of the chunk two before, which the warps release after their x pass. It follows
  // the chunk it computes by one
  int64_t p_task = blockIdx.x;
  int p_ch = 0;
  uint32_t issued = 0;
  auto issue = [&]() -> bool {
    if (p_task >= ntask) return true;
    const int st = (int)(issued & 1);
    int good = 1;
    if (lane == 0) {
      if (issued >= 2) good = mbar_wait(&empty[st], ((issued >> 1) - 1) & 1u, p.timeout_ns, p.status);
      if (good) mbar_arrive_expect_tx(&full[st], (uint32_t)(nband * bandsz * 16));
    }
    if (!__shfl_sync(0xffffffffu, good, 0)) return false;
    if (lane < nband) {
      const int z = (int)(p_task / per_z);
      int64_t r = p_task - z * per_z;
      const int kl = (int)(r / ((int64_t)p.ga * p.gb));
      r -= (int64_t)kl * p.ga * p.gb;
      const int a0 = (int)(r / p.gb) * p.na, b0 = (int)(r % p.gb) * p.nb;
      // bands past the end repeat the last one; their pairs are not stored
      const int64_t band = lane < p.na ? (int64_t)kl * p.nocc + min(a0 + lane, p.nocc - 1)
                                       : (int64_t)kl * p.nunocc + min(b0 + lane - p.na, p.nunocc - 1);
      const double2* src = (lane < p.na ? p.A : p.B) + (band * p.n + z) * p.n * p.ld;
      double2* dst = stage + ((size_t)st * nband + lane) * bandsz;
      const uint32_t line = (uint32_t)p.ld * 16;
      const int y0 = p_ch * FFS_SLOTS;
      bulk_g2s(dst, src + (int64_t)y0 * p.ld, 8 * line, &full[st]);
      // mirrors of slots 7 .. 1 are the lines n - y0 - 7 .. n - y0 - 1, that of slot 0 is the
      // next one, or for y = 0 the line n / 2
      bulk_g2s(dst + 8 * p.ld, src + (int64_t)(p.n - y0 - 7) * p.ld, 7 * line, &full[st]);
      bulk_g2s(dst + 15 * p.ld, src + (int64_t)(y0 ? p.n - y0 : p.n / 2) * p.ld, line, &full[st]);
    }
    ++issued;
    if (++p_ch == p.nst) p_ch = 0, p_task += gridDim.x;
    return true;
  };
  // leave after a wait ran out: copies still landing must finish before this CTA's shared
  // memory goes away
  auto give_up = [&](uint32_t c) {
    if (warp == 0 && lane == 0)
      for (uint32_t k = c; k < issued; ++k) mbar_drain(&full[k & 1], (k >> 1) & 1u, p.timeout_ns);
  };
  if (warp == 0) issue();   // (the first two chunks wait for nothing)

  const int g = lane >> 2, t = lane & 3;
  const int ia = warp / p.nb, ib = warp % p.nb;
  const bool even = (p.n & 1) == 0;
  const double alt = t ? 0.0 : ((g & 1) ? -1.0 : 1.0);   // A fragment of the point n / 2: (-1)^k at slot 0
  const int row[2] = {g * p.ld, (15 - g) * p.ld};         // this thread's line and its mirror
  const double2* wt = tab + g * p.sl;
  uint32_t c = 0;
  for (int64_t task = blockIdx.x; task < ntask; task += gridDim.x) {
    // [C re, C im, S re, S im of the x pass][cos, sin][ky = g, kx = 2t + e]
    double ya[4][2][2];
#pragma unroll
    for (int x = 0; x < 4; ++x) ya[x][0][0] = ya[x][0][1] = ya[x][1][0] = ya[x][1][1] = 0.0;
    for (int ch = 0; ch < p.nst; ++ch, ++c) {
      const int st = (int)(c & 1);
      if ((warp == 0 && !issue()) || !mbar_wait(&full[st], (c >> 1) & 1u, p.timeout_ns, p.status)) {
        give_up(c);
        return;
      }
      const double2* sa = stage + ((size_t)st * nband + ia) * bandsz;
      const double2* sb = stage + ((size_t)st * nband + p.na + ib) * bandsz;
      // x pass: [line, mirror][C re, C im, S re, S im][kx = g, lines 2t + e]
      double za[2][4][2];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int x = 0; x < 4; ++x) za[h][x][0] = za[h][x][1] = 0.0;
#pragma unroll 2
      for (int s = 0; s < 2 * p.nst; ++s) {
        const int zi = 4 * s + t, zm = zi ? p.n - zi : 0;
        const double2 w = wt[zi];
        double f[2][4];   // folded products of line g at slot zi: c re, c im, s re, s im
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double2 a = sa[row[h] + zi];
          double2 am = sa[row[h] + zm];
          if (zi == 0) am = make_double2(0.0, 0.0);
          const double2 u = cmul(a, sb[row[h] + zi]), v = cmul(am, sb[row[h] + zm]);
          f[h][0] = u.x + v.x;
          f[h][1] = u.y + v.y;
          f[h][2] = u.x - v.x;
          f[h][3] = u.y - v.y;
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int h = 0; h < 2; ++h) dmma_8x8x4(za[h][x], x < 2 ? w.x : w.y, f[h][x]);
      }
      if (even) {
        // the self-paired point n / 2 of every line
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double2 u = cmul(sa[row[h] + p.n / 2], sb[row[h] + p.n / 2]);
          dmma_8x8x4(za[h][0], alt, t ? 0.0 : u.x);
          dmma_8x8x4(za[h][1], alt, t ? 0.0 : u.y);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[st]);

      // y pass: slots y = 2t + e, folded with their mirrors; that of y = 0 is the line n / 2
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int y = ch * FFS_SLOTS + 2 * t + e;
        const double2 w = wt[y];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const double a = za[0][x][e], m = y ? za[1][x][e] : 0.0;
          const double u = y < p.H ? a + m : 0.0, v = y < p.H ? a - m : 0.0;
          dmma_8x8x4(ya[x][0], w.x, u);
          dmma_8x8x4(ya[x][1], w.y, v);
        }
      }
      if (even && ch == 0) {
#pragma unroll
        for (int x = 0; x < 4; ++x) dmma_8x8x4(ya[x][0], alt, t ? 0.0 : za[1][x][0]);
      }
    }

    // outputs of (+-kx, +-ky), ky = g, kx = 2t + e
    const int z = (int)(task / per_z);
    int64_t r = task - z * per_z;
    const int kl = (int)(r / ((int64_t)p.ga * p.gb));
    r -= (int64_t)kl * p.ga * p.gb;
    const int n1 = (int)(r / p.gb) * p.na + ia, n2 = (int)(r % p.gb) * p.nb + ib;
    const int py[2] = {pos[16 + 7 + g], g ? pos[16 + 7 - g] : -1};
    if (n1 >= p.nocc || n2 >= p.nunocc) continue;
    const int64_t pair = ((int64_t)kl * p.nocc + n1) * p.nunocc + n2;
    double2* out = p.T2 + (pair * p.n + z) * p.nkx * p.nky;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int kx = 2 * t + e;
      const int px[2] = {pos[7 + kx], kx ? pos[7 - kx] : -1};
      // y transform of the C and of the S sequence: cosine and sine sums
      const double2 cc = make_double2(ya[0][0][e], ya[1][0][e]), cs = make_double2(ya[0][1][e], ya[1][1][e]);
      const double2 sc = make_double2(ya[2][0][e], ya[3][0][e]), ss = make_double2(ya[2][1][e], ya[3][1][e]);
#pragma unroll
      for (int my = 0; my < 2; ++my) {
        if (py[my] < 0) continue;
        const double2 C = my ? fold_minus(cc, cs) : fold_plus(cc, cs);
        const double2 S = my ? fold_minus(sc, ss) : fold_plus(sc, ss);
        if (px[0] >= 0) out[px[0] * p.nky + py[my]] = fold_plus(C, S);
        if (px[1] >= 0) out[px[1] * p.nky + py[my]] = fold_minus(C, S);
      }
    }
  }
}

struct FoldGatherParams {
  const double2* T2;   // [pair][z][kx][ky]
  const double2* tab;  // as FoldParams
  const int* posz;
  const int* gmap;     // per ig: iz | iy << 8 | ix << 16
  double2* cprod;      // (first pair of the chunk, column col0)
  int64_t ldc, npair;
  int n, nst, sl, nkz, plane, nky, ngptm;
};

// The z pass and the gather: a CTA takes two consecutive pairs (32-byte runs of a cprod
// column); its 8 warps share their 16-line row blocks. Every value of T2 is read once, in
// 128-byte runs, straight into the folded fragments; the spectra of the two pairs meet in
// shared memory. Measured at 24000 pairs, 13^2 lines of 48: 3.65 ms summed per vector on the
// CUDA cores, 1.06 ms here (3.1 GB of T2, 0.8 GB of cprod).
__global__ void __launch_bounds__(256) fft_pair_gather_kernel(FoldGatherParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double2* F = reinterpret_cast<double2*>(smem_raw);          // [2][nkz][plane]
  double2* tab = F + 2 * (size_t)p.nkz * p.plane;             // [8][sl]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  for (int i = threadIdx.x; i < FFS_K * p.sl; i += blockDim.x) tab[i] = p.tab[i];
  __syncthreads();
  const int64_t pair0 = 2 * (int64_t)blockIdx.x;
  const int np = (int)min((int64_t)2, p.npair - pair0);
  const int nrb = (p.plane + FFS_ROWS - 1) / FFS_ROWS;
  const bool even = (p.n & 1) == 0;
  for (int it = warp; it < np * nrb; it += 8) {
    const int pr = it / nrb, l0 = (it - pr * nrb) * FFS_ROWS;
    const double2* src = p.T2 + (pair0 + pr) * p.n * p.plane;
    int line[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) line[h] = min(l0 + g + 8 * h, p.plane - 1);
    double za[4][4];
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int r = 0; r < 4; ++r) za[x][r] = 0.0;
#pragma unroll 1
    for (int s = 0; s < p.nst; ++s) {
      double2 w[2], v[2][2], vm[2][2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int zi = 8 * s + t + 4 * q, zm = zi ? p.n - zi : 0;
        w[q] = tab[g * p.sl + zi];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          v[q][h] = __ldg(src + (int64_t)zi * p.plane + line[h]);
          vm[q][h] = __ldg(src + (int64_t)zm * p.plane + line[h]);
          if (zi == 0) vm[q][h] = make_double2(0.0, 0.0);
        }
      }
      double f[4][4];
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          f[0][2 * q + h] = v[q][h].x + vm[q][h].x;
          f[1][2 * q + h] = v[q][h].y + vm[q][h].y;
          f[2][2 * q + h] = v[q][h].x - vm[q][h].x;
          f[3][2 * q + h] = v[q][h].y - vm[q][h].y;
        }
      const double wc[2] = {w[0].x, w[1].x}, ws[2] = {w[0].y, w[1].y};
#pragma unroll
      for (int x = 0; x < 4; ++x) dmma_16x8x8(za[x], f[x], x < 2 ? wc : ws);
    }
    double2* Fp = F + (size_t)pr * p.nkz * p.plane;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (even) {
        const double2 u = __ldg(src + (int64_t)(p.n / 2) * p.plane + line[h]);
        za[0][2 * h] += u.x;
        za[0][2 * h + 1] -= u.x;
        za[1][2 * h] += u.y;
        za[1][2 * h + 1] -= u.y;
      }
      if (l0 + g + 8 * h >= p.plane) continue;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int kz = 2 * t + e, r = 2 * h + e;
        const double2 C = make_double2(za[0][r], za[1][r]), S = make_double2(za[2][r], za[3][r]);
        const int ip = p.posz[7 + kz], im = kz ? p.posz[7 - kz] : -1;
        if (ip >= 0) Fp[ip * p.plane + line[h]] = fold_plus(C, S);
        if (im >= 0) Fp[im * p.plane + line[h]] = fold_minus(C, S);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < np * p.ngptm; i += blockDim.x) {
    const int ig = i / np, pr = i - ig * np, m = p.gmap[ig];
    const int iz = m & 255, iy = (m >> 8) & 255, ix = (m >> 16) & 255;
    const double2 v = F[((size_t)pr * p.nkz + iz) * p.plane + ix * p.nky + iy];
    double2* o = p.cprod + pair0 + pr + p.ldc * ig;
    double2 u = *o;
    u.x += v.x;
    u.y += v.y;
    *o = u;
  }
}

// ---------------------------------------------------------------------------
// host

struct Box3 {
  int lo[3] = {0, 0, 0}, dim[3] = {1, 1, 1};
  int64_t size() const { return (int64_t)dim[0] * dim[1] * dim[2]; }
};

static Box3 box_of(const int* g, int n) {
  Box3 b;
  if (n == 0) return b;
  int hi[3];
  for (int c = 0; c < 3; ++c) b.lo[c] = hi[c] = g[c];
  for (int i = 0; i < n; ++i)
    for (int c = 0; c < 3; ++c) {
      b.lo[c] = std::min(b.lo[c], g[3 * i + c]);
      hi[c] = std::max(hi[c], g[3 * i + c]);
    }
  for (int c = 0; c < 3; ++c) b.dim[c] = hi[c] - b.lo[c] + 1;
  return b;
}

struct FftPlan {
  int n = 0;
  Box3 b1, b2, bs;
  std::vector<int> gidx1, gidx2, ks[3], gmap;
  std::vector<double2> twb, twf;
  // the folded passes: every component of G_M within 7 of the origin modulo n
  bool sym = false;
  int ld = 0, H = 0, nst = 0, sl = 0;
  std::vector<int> pos[3];       // index of k in ks[c] at k + 7, or -1
  std::vector<double2> tab;      // FoldParams::tab
};

// |k| <= 7 for the residue v of k modulo n, as k itself; 99 otherwise.
static int fold_k(int v, int n) {
  const int k = v > n / 2 ? v - n : v;
  return k >= -7 && k <= 7 ? k : 99;
}

// fold: whether the folded passes may be taken (their padded lines need a little more scratch).
static int plan_fft(spx_ctx* ctx, const spx_pw_desc* d, FftPlan* pl, bool fold = true) {
  const int n = d->nfft;
  if (n < 2 || n > FFT_NMAX)
    return set_error(ctx, SPX_EINVAL, "nfft must be in 2..64 for the FFT branch");
  if (d->ngptm > 4096) return set_error(ctx, SPX_EINVAL, "FFT branch supports ngptm <= 4096");
  if (d->step_radius < 0 || d->step_radius > 4 || d->vol <= 0.0)
    return set_error(ctx, SPX_EINVAL, "bad plane-wave descriptor (step_radius must be 0..4)");
  if ((d->ngpt1 > 0 && !d->gpt1) || (d->ngpt2 > 0 && !d->gpt2) || (d->ngptm > 0 && !d->gptm) || !d->cstep)
    return set_error(ctx, SPX_EINVAL, "null plane-wave descriptor array");
  pl->n = n;
  pl->b1 = box_of(d->gpt1, d->ngpt1);
  pl->b2 = box_of(d->gpt2, d->ngpt2);
  // G_M alone within 7 of the origin on every axis: the folded passes, with the backfolding
  // vector in the step function (exp(2 pi i g r / n) theta(r) shifts the product's spectrum)
  pl->sym = fold && n >= 16;
  for (int i = 0; i < 3 * d->ngptm && pl->sym; ++i)
    pl->sym = fold_k(((d->gptm[i] % n) + n) % n, n) != 99;
  for (int c = 0; c < 3; ++c) {
    pl->bs.lo[c] = -d->step_radius + (pl->sym ? d->gshift[c] : 0);
    pl->bs.dim[c] = 2 * d->step_radius + 1;
  }
  auto lin = [](const Box3& b, const int* g) {
    return (int)((g[0] - b.lo[0]) + (int64_t)b.dim[0] * ((g[1] - b.lo[1]) + (int64_t)b.dim[1] * (g[2] - b.lo[2])));
  };
  if (pl->b1.size() > (1 << 26) || pl->b2.size() > (1 << 26))
    return set_error(ctx, SPX_EINVAL, "plane-wave G boxes too large");
  pl->gidx1.resize(d->ngpt1);
  for (int i = 0; i < d->ngpt1; ++i) pl->gidx1[i] = lin(pl->b1, d->gpt1 + 3 * i);
  pl->gidx2.resize(d->ngpt2);
  for (int i = 0; i < d->ngpt2; ++i) pl->gidx2[i] = lin(pl->b2, d->gpt2 + 3 * i);
  // distinct (G_M - g) mod n (G_M mod n with g in the step function) per axis, and each
  // ig's position in them
  std::vector<int> idx[3];
  for (int c = 0; c < 3; ++c) {
    std::vector<int> v(d->ngptm);
    for (int i = 0; i < d->ngptm; ++i) v[i] = (((d->gptm[3 * i + c] - (pl->sym ? 0 : d->gshift[c])) % n) + n) % n;
    pl->ks[c] = v;
    std::sort(pl->ks[c].begin(), pl->ks[c].end());
    pl->ks[c].erase(std::unique(pl->ks[c].begin(), pl->ks[c].end()), pl->ks[c].end());
    if ((int)pl->ks[c].size() > FFT_KMAX)
      return set_error(ctx, SPX_ENOTSUP,
                       "FFT branch: more than 16 distinct mixed-basis G components per axis; "
                       "use the explicit convolution (nfft = 0)");
    idx[c].resize(d->ngptm);
    for (int i = 0; i < d->ngptm; ++i)
      idx[c][i] = (int)(std::lower_bound(pl->ks[c].begin(), pl->ks[c].end(), v[i]) - pl->ks[c].begin());
  }
  pl->gmap.resize(d->ngptm);
  for (int i = 0; i < d->ngptm; ++i) pl->gmap[i] = idx[2][i] | (idx[1][i] << 8) | (idx[0][i] << 16);
  pl->twb.resize(n);
  pl->twf.resize(n);
  for (int m = 0; m < n; ++m) {
    const long double ang = 2.0L * 3.14159265358979323846264338327950288L * m / n;
    const double c = (double)cosl(ang), s = (double)sinl(ang);
    pl->twb[m] = make_double2(c, s);
    pl->twf[m] = make_double2(c, -s);
  }
  pl->ld = n;
  if (pl->sym) {
    // rows of 4 (mod 8) elements: consecutive lines start in different halves of the banks
    pl->ld = n + (12 - n % 8) % 8;
    pl->H = (n + 1) / 2;
    pl->nst = (pl->H + FFS_SLOTS - 1) / FFS_SLOTS;
    pl->sl = FFS_SLOTS * pl->nst + 4;
    pl->tab.assign((size_t)FFS_K * pl->sl, make_double2(0.0, 0.0));
    for (int k = 0; k < FFS_K; ++k)
      for (int z = 0; z < pl->H; ++z) {
        const double2 w = pl->twb[(k * z) % n];
        pl->tab[(size_t)k * pl->sl + z] = w;
      }
    for (int c = 0; c < 3; ++c) {
      pl->pos[c].assign(15, -1);
      for (size_t i = 0; i < pl->ks[c].size(); ++i) pl->pos[c][fold_k(pl->ks[c][i], n) + 7] = (int)i;
    }
  }
  return SPX_OK;
}

// Scratch of a call: the plan's tables, copied as one block; theta(r); and for `kchunk` k points
// the band grids A and B and one region that first holds the passes' buffers (box, ta, tb), then
// T2, which is written after the last of them has run.
struct FftScratch {
  size_t o_g1, o_g2, o_ks[3], o_gmap, o_twb, o_twf, o_cs, o_pos[3], o_tab, tables;   // bytes
  size_t box, ta, tb, A, B, T2;   // elements per k point
  size_t theta, theta_ta, theta_tb;
  FftScratch() = default;
  FftScratch(const FftPlan& pl, const spx_pw_desc* d, int nocc, int nunocc) {
    const size_t n = (size_t)pl.n, nb = (size_t)std::max(nocc, nunocc), n2ld = n * n * (size_t)pl.ld;
    size_t at = 0;
    auto table = [&](size_t bytes) {
      const size_t o = at;
      at += align_up(std::max<size_t>(bytes, 1), 256);
      return o;
    };
    o_g1 = table(4 * (size_t)d->ngpt1);
    o_g2 = table(4 * (size_t)d->ngpt2);
    for (int c = 0; c < 3; ++c) o_ks[c] = table(4 * pl.ks[c].size());
    o_gmap = table(4 * (size_t)d->ngptm);
    o_twb = table(16 * n);
    o_twf = table(16 * n);
    o_cs = table(16 * (size_t)pl.bs.size());
    for (int c = 0; c < 3; ++c) o_pos[c] = table(4 * pl.pos[c].size());
    o_tab = table(16 * pl.tab.size());
    tables = at;
    box = nb * (size_t)std::max(pl.b1.size(), pl.b2.size());
    ta = nb * n * (size_t)std::max(pl.b1.dim[1] * pl.b1.dim[2], pl.b2.dim[1] * pl.b2.dim[2]);
    tb = nb * n * n * (size_t)std::max(pl.b1.dim[2], pl.b2.dim[2]);
    A = (size_t)nocc * n2ld;
    B = (size_t)nunocc * n2ld;
    T2 = (size_t)nocc * (size_t)nunocc * n * pl.ks[0].size() * pl.ks[1].size();
    theta = n * n * n;
    theta_ta = n * (size_t)(pl.bs.dim[1] * pl.bs.dim[2]);
    theta_tb = n * n * (size_t)pl.bs.dim[2];
  }
  size_t passes(size_t k) const {   // of the region: buffers of k k points, or of theta
    return align_up(16 * k * box, 256) + align_up(16 * std::max(k * ta, theta_ta), 256) +
           align_up(16 * std::max(k * tb, theta_tb), 256);
  }
  size_t region(size_t k) const { return std::max(align_up(16 * k * T2, 256), passes(k)); }
  size_t bytes(size_t k) const {
    return tables + align_up(16 * theta, 256) + align_up(16 * k * A, 256) + align_up(16 * k * B, 256) + region(k);
  }
  // Most k points, up to nk and at least one, within `left` bytes.
  int kchunk(int nk, size_t left) const {
    int lo = 1, hi = nk;
    while (lo < hi) {
      const int mid = lo + (hi - lo + 1) / 2;
      if (bytes((size_t)mid) <= left) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  }
};

// The plan and scratch of a call within `room` bytes: folded passes where they fit.
static int fft_plan_within(spx_ctx* ctx, const spx_pw_desc* d, int nocc, int nunocc, size_t room, FftPlan* pl,
                           FftScratch* sc) {
  int rc = plan_fft(ctx, d, pl);
  if (rc) return rc;
  *sc = FftScratch(*pl, d, nocc, nunocc);
  if (!pl->sym || sc->bytes(1) <= room) return SPX_OK;
  *pl = FftPlan();
  if ((rc = plan_fft(ctx, d, pl, false))) return rc;
  *sc = FftScratch(*pl, d, nocc, nunocc);
  return SPX_OK;
}

// room: the most the caller can have, 0 = no limit.
size_t wfprod_pw_fft_workspace(const spx_pw_desc* d, int nk, int nocc, int nunocc, size_t room) {
  spx_ctx dummy;
  FftPlan pl;
  FftScratch sc;
  const size_t most = room ? room - std::min<size_t>(room, 256) : SIZE_MAX;
  if (fft_plan_within(&dummy, d, nocc, nunocc, most, &pl, &sc)) return 0;
  return sc.bytes((size_t)sc.kchunk(std::max(nk, 1), std::min(most, (size_t)6 << 30))) + 256;
}

// Three passes G box -> r grid for nb bands: box [b][gz][gy][gx] -> out [b][z][y][ld].
static int band_grids(spx_ctx* ctx, const Box3& bx, int nb, const double2* box, double2* ta,
                      double2* tb, double2* out, int ld, const double2* twb, int n, int conj_out,
                      double scale, const double2* mul, cudaStream_t s, int* launches) {
  if (nb == 0) return SPX_OK;
  const int64_t X = bx.dim[0], Y = bx.dim[1], Z = bx.dim[2], nh = n / 2 + 1;
  auto grid_for = [&](int64_t total) {
    return (unsigned)std::min<int64_t>((total + 255) / 256, (int64_t)ctx->num_sms * 32);
  };
  // x: box[b][gz][gy][gx] -> ta[b][gz][gy][x]
  const int64_t nline = nb * Z * Y;
  dft_line_kernel<<<grid_for(nline * nh), 256, 0, s>>>(box, ta, twb, (int)X, bx.lo[0], n, nline);
  const int64_t ng = (nh + DFT_JP - 1) / DFT_JP;
  DftAcross p{};
  p.tw = twb;
  p.n = n;
  p.scale = 1.0;
  // y: ta[b][gz][gy][x] -> tb[b][gz][y][x]
  p.in = ta; p.out = tb; p.nin = (int)Y; p.lo = bx.lo[1]; p.n2 = 1; p.outer = nb * Z;
  p.is = n; p.i1 = Y * n; p.sj = n; p.s1 = (int64_t)n * n;
  dft_across_kernel<<<grid_for(p.outer * ng * n), 256, 0, s>>>(p);
  // z: tb[b][gz][y][x] -> out[b][z][y][x], with the post-operation
  p.in = tb; p.out = out; p.nin = (int)Z; p.lo = bx.lo[2]; p.n2 = n; p.outer = (int64_t)nb * n;
  p.is = (int64_t)n * n; p.i1 = Z * n * n; p.i2 = n;
  p.sj = (int64_t)n * ld; p.s1 = (int64_t)n * n * ld; p.s2 = ld;
  p.conj_out = conj_out; p.scale = scale; p.mul = mul; p.mj = (int64_t)n * n; p.m2 = n;
  dft_across_kernel<<<grid_for(p.outer * ng * n), 256, 0, s>>>(p);
  *launches += 3;
  return check_cuda(ctx, cudaGetLastError(), "band grid passes");
}

int wfprod_pw_fft_run(spx_ctx* ctx, const spx_pw_desc* d, int nk, int nocc, int nunocc,
                      const double2* c1, const double2* c2, double2* cprod, int64_t ldc, int col0,
                      void* ws, size_t ws_bytes, cudaStream_t s, int* launches) {
  FftPlan pl;
  FftScratch sc;
  char* base = (char*)align_up((size_t)ws, 256);
  const size_t left = ws_bytes - std::min(ws_bytes, (size_t)(base - (char*)ws));
  int rc = fft_plan_within(ctx, d, nocc, nunocc, left, &pl, &sc);
  if (rc) return rc;
  if (d->ngptm == 0 || nk == 0 || nocc == 0 || nunocc == 0 || !ws) return SPX_OK;
  if ((nunocc + FFT_NP - 1) / FFT_NP > 65535)
    return set_error(ctx, SPX_EINVAL, "too many unoccupied bands for the FFT branch");
  const int n = pl.n, nkx = (int)pl.ks[0].size(), nky = (int)pl.ks[1].size(), nkz = (int)pl.ks[2].size();
  const int64_t n3 = (int64_t)n * n * n;
  if (left < sc.bytes(1)) return set_error(ctx, SPX_ENOMEM, "FFT-branch scratch too small");
  // grid limit of K5c: one CTA per pair of a chunk along x
  const size_t pairs_k = (size_t)nocc * nunocc;
  if (pairs_k > 2147483647u) return set_error(ctx, SPX_EINVAL, "too many band pairs per k point");
  const int kchunk = std::min(sc.kchunk(nk, left), (int)std::min<size_t>((size_t)nk, 2147483647u / pairs_k));
  const size_t kc = (size_t)kchunk;
  auto at = [&](size_t o) { return base + o; };
  const int *d_g1 = (int*)at(sc.o_g1), *d_g2 = (int*)at(sc.o_g2), *d_gmap = (int*)at(sc.o_gmap);
  const int *d_ks[3], *d_pos[3];
  for (int c = 0; c < 3; ++c) d_ks[c] = (int*)at(sc.o_ks[c]), d_pos[c] = (int*)at(sc.o_pos[c]);
  const double2 *d_twb = (double2*)at(sc.o_twb), *d_twf = (double2*)at(sc.o_twf), *d_cs = (double2*)at(sc.o_cs),
                *d_tab = (double2*)at(sc.o_tab);
  double2* theta = (double2*)at(sc.tables);
  double2* A = (double2*)((char*)theta + align_up(16 * sc.theta, 256));
  double2* Bg = (double2*)((char*)A + align_up(16 * kc * sc.A, 256));
  double2* T2 = (double2*)((char*)Bg + align_up(16 * kc * sc.B, 256));
  double2* box = T2;
  double2* ta = (double2*)((char*)box + align_up(16 * kc * sc.box, 256));
  double2* tb = (double2*)((char*)ta + align_up(16 * std::max(kc * sc.ta, sc.theta_ta), 256));
  // the tables in one copy: small calls are bound by the host's launches and copies
  std::vector<char> tables(sc.tables);
  auto put = [&](size_t o, const void* src, size_t bytes) {
    if (bytes) std::memcpy(tables.data() + o, src, bytes);
  };
  put(sc.o_g1, pl.gidx1.data(), 4 * pl.gidx1.size());
  put(sc.o_g2, pl.gidx2.data(), 4 * pl.gidx2.size());
  for (int c = 0; c < 3; ++c) {
    put(sc.o_ks[c], pl.ks[c].data(), 4 * pl.ks[c].size());
    put(sc.o_pos[c], pl.pos[c].data(), 4 * pl.pos[c].size());
  }
  put(sc.o_gmap, pl.gmap.data(), 4 * pl.gmap.size());
  put(sc.o_twb, pl.twb.data(), 16 * (size_t)n);
  put(sc.o_twf, pl.twf.data(), 16 * (size_t)n);
  put(sc.o_cs, d->cstep, 16 * (size_t)pl.bs.size());
  put(sc.o_tab, pl.tab.data(), 16 * pl.tab.size());
  if ((rc = check_cuda(ctx, cudaMemcpyAsync(base, tables.data(), sc.tables, cudaMemcpyHostToDevice, s), "copy plan")) ||
      (rc = check_cuda(ctx, cudaStreamSynchronize(s), "copy plan")))
    return rc;
  // theta(r) from the step-function box (already laid out x fastest)
  if ((rc = band_grids(ctx, pl.bs, 1, d_cs, ta, tb, theta, n, d_twb, n, 0, 1.0, nullptr, s, launches)))
    return rc;
  const size_t zy_smem = sizeof(double2) * ((size_t)n * n + 2 * FFT_KMAX * n + (size_t)FFT_NP * FFT_KMAX * n);
  const size_t x_smem = sizeof(double2) * ((size_t)FFT_KMAX * n + d->ngptm + (size_t)FFT_XC * nkx * nky);
  cudaFuncSetAttribute(fft_pair_zy_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zy_smem);
  // grid edges 16 r (r <= 4) take the line FFT; bpc bands per CTA within 108 KB of
  // shared memory and 512 threads
  const bool radix = !pl.sym && n % 16 == 0 && n / 16 >= 1 && n / 16 <= 4;
  const size_t band_smem = sizeof(double2) * ((size_t)n * (n / 16) * FFTR_LD + (size_t)FFT_KMAX * (n + 1));
  const int bpc = radix ? std::max(1, std::min({4, 512 / (n * (n / 16)), (int)((108 << 10) / band_smem)})) : 1;
  const size_t radix_smem = sizeof(double2) * ((size_t)n + 16) + bpc * band_smem;
  if (radix)
    cudaFuncSetAttribute(fft_pair_zy_radix_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)radix_smem);
  cudaFuncSetAttribute(fft_pair_x_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)x_smem);
  // folded passes: 4 x 4 bands per CTA, or 2 x 4 where two stages of eight bands do not fit
  // (grid edges above 48)
  auto fold_smem = [&](int na, int nb) {
    return sizeof(double2) * ((size_t)2 * (na + nb) * FFS_ROWS * pl.ld + (size_t)FFS_K * pl.sl) +
           4 * sizeof(uint64_t) + 32 * sizeof(int);
  };
  const int fna = fold_smem(4, 4) <= (227 << 10) ? 4 : 2, fnb = 4;
  const size_t f_smem = fold_smem(fna, fnb);
  const size_t g_smem = sizeof(double2) * ((size_t)2 * nkz * nkx * nky + (size_t)FFS_K * pl.sl);
  if (pl.sym && ((rc = check_cuda(ctx, cudaFuncSetAttribute(fft_pair_fold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                            (int)f_smem), "fold attribute")) ||
                 (rc = check_cuda(ctx, cudaFuncSetAttribute(fft_pair_gather_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                            (int)g_smem), "gather attribute"))))
    return rc;
  for (int k0 = 0; k0 < nk; k0 += kchunk) {
    const int kn = std::min(kchunk, nk - k0);
    // occupied: conj(phi)/sqrt(vol) * theta; unoccupied: phi / nnfft
    const int nb1 = kn * nocc, nb2 = kn * nunocc;
    if ((rc = check_cuda(ctx, cudaMemsetAsync(box, 0, 16 * (size_t)nb1 * pl.b1.size(), s), "zero box"))) return rc;
    if (d->ngpt1 > 0) {
      dim3 g((d->ngpt1 + 255) / 256, nb1);
      fft_scatter_kernel<<<g, 256, 0, s>>>(c1 + (int64_t)k0 * nocc * d->ngpt1, d->ngpt1, d_g1, pl.b1.size(), box);
      ++*launches;
    }
    if ((rc = band_grids(ctx, pl.b1, nb1, box, ta, tb, A, pl.ld, d_twb, n, 1, 1.0 / std::sqrt(d->vol), theta, s, launches)))
      return rc;
    if ((rc = check_cuda(ctx, cudaMemsetAsync(box, 0, 16 * (size_t)nb2 * pl.b2.size(), s), "zero box"))) return rc;
    if (d->ngpt2 > 0) {
      dim3 g((d->ngpt2 + 255) / 256, nb2);
      fft_scatter_kernel<<<g, 256, 0, s>>>(c2 + (int64_t)k0 * nunocc * d->ngpt2, d->ngpt2, d_g2, pl.b2.size(), box);
      ++*launches;
    }
    if ((rc = band_grids(ctx, pl.b2, nb2, box, ta, tb, Bg, pl.ld, d_twb, n, 0, 1.0 / (double)n3, nullptr, s, launches)))
      return rc;
    if (pl.sym) {
      FoldParams fp{A, Bg, T2, d_tab, d_pos[0], d_pos[1], n, pl.ld, pl.H, pl.nst, pl.sl, kn, nocc, nunocc, fna, fnb,
                    nkx, nky, (nocc + fna - 1) / fna, (nunocc + fnb - 1) / fnb, ctx->d_status,
                    (uint64_t)(ctx->opt.timeout_ms > 0 ? ctx->opt.timeout_ms : 4000) * 1000000ull};
      const int64_t ntask = (int64_t)kn * fp.ga * fp.gb * n;
      fft_pair_fold_kernel<<<(unsigned)std::min<int64_t>(ntask, ctx->num_sms), 32 * fna * fnb, f_smem, s>>>(fp);
      if ((rc = check_cuda(ctx, cudaGetLastError(), "fft_pair_fold_kernel launch"))) return rc;
      const int64_t npair = (int64_t)kn * nocc * nunocc;
      FoldGatherParams gp{T2, d_tab, d_pos[2], d_gmap, cprod + (int64_t)k0 * nocc * nunocc + ldc * col0, ldc, npair,
                          n, pl.nst, pl.sl, nkz, nkx * nky, nky, d->ngptm};
      fft_pair_gather_kernel<<<(unsigned)((npair + 1) / 2), 256, g_smem, s>>>(gp);
      if ((rc = check_cuda(ctx, cudaGetLastError(), "fft_pair_gather_kernel launch"))) return rc;
      *launches += 2;
      continue;
    }
    if (radix) {
      PairFftParams pr{A, Bg, T2, d_twf, d_ks[0], d_ks[1], n, n / 16, bpc, nocc, nunocc, nkx, nky};
      dim3 gz(nb1, (nunocc + bpc - 1) / bpc, n);
      fft_pair_zy_radix_kernel<<<gz, bpc * n * (n / 16), radix_smem, s>>>(pr);
      if ((rc = check_cuda(ctx, cudaGetLastError(), "fft_pair_zy_radix_kernel launch"))) return rc;
    } else {
      PairParams pp{A, Bg, T2, d_twf, d_ks[0], d_ks[1], n, nocc, nunocc, nkx, nky};
      dim3 gz(nb1, (nunocc + FFT_NP - 1) / FFT_NP, n), bz(n, FFT_NP);
      fft_pair_zy_kernel<<<gz, bz, zy_smem, s>>>(pp);
      if ((rc = check_cuda(ctx, cudaGetLastError(), "fft_pair_zy_kernel launch"))) return rc;
    }
    ++*launches;
    // (the kernel's x is the plane axis z, its z the line axis x)
    GatherParams gp{T2, d_twf, d_ks[2], d_gmap, cprod + (int64_t)k0 * nocc * nunocc + ldc * col0, ldc,
                    n, nkz, nky, nkx, d->ngptm};
    fft_pair_x_kernel<<<(unsigned)((int64_t)kn * nocc * nunocc), 256, x_smem, s>>>(gp);
    if ((rc = check_cuda(ctx, cudaGetLastError(), "fft_pair_x_kernel launch"))) return rc;
    ++*launches;
  }
  return SPX_OK;
}

}  // namespace spx
