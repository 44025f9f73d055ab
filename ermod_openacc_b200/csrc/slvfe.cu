// slvfe.cu -- slvfe's free-energy functional (chmpot) for one data set on the GPU, in FP64,
// with slvfe's default options (sfemain.F90:22-64): py-hnc, regularised Cholesky solve of
// the reference-solvent equation, eczr zero shift, harmonic extrapolation weights, linear
// extrapolation of omega in solution, normalize 'yes', no bin merging.
//
//   k_slv_prep     distnorm's per-species scaling of rho / rho0 (slvfe.F90:1467-1502) and
//                  omega in solution where both distributions are sampled (getslncv :875-930)
//   k_slv_colsum, k_slv_sweep, k_slv_scale
//                  the chi0 row scaling (slvfe.F90:1503-1525): Gauss-Seidel sweeps over the
//                  bins, each bin's correction from the corrections already updated in this
//                  sweep, to 1e-8 within 100 sweeps
//   k_slv_extrap   omega in solution for bins sampled on one side only (:930-1001): a
//                  weighted linear fit over the species' sampled bins, a thread per bin
//   k_slv_reg      the per-species regularisation trace / count^2 (getinscv :1003-1120)
//   k_slv_build    A = chi0 - rho0 rho0^T (+ reg per species block, 1 on unsampled
//                  diagonals), padded to a multiple of the tile with the identity
//   k_chol_first, k_chol_step, k_slv_back
//                  blocked right-looking Cholesky of A (32 x 32 FP64 tiles, one launch a step)
//                  with the forward substitution carried along, and the backward substitution
//   k_slv_check    posv_wrap's acceptance of that solution (slvfe.F90:520-531): the
//                  largest residual against the regularised matrix, the largest element
//   eigen-decomposition fallback (getinscv :1124-1170), when the Cholesky factor fails
//   or the check rejects the solution: the unregularised matrix (k_slv_unreg) goes to
//   cuSOLVER's Dsyevd, as the reference's syevr_wrap sends it to cusolverDnSsyevd; its
//   first nsp eigenpairs are skipped in the pseudo-inverse (k_slv_evd_coef, k_slv_evd_x)
//   k_slv_chmpot   the eczr zero shift, the functional and its per-species sums (:744-803)
//
// Every reduction is a fixed-order tree, so a run is reproducible bit for bit.
#include <cuda_runtime.h>
#include <cusolverDn.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/ermod_slvfe.h"
#include "workspace.cuh"

namespace erm {
cudaError_t staged_to_device(void* dst, const void* src, size_t bytes, cudaStream_t s);   // staging.cu
}

namespace {

constexpr int kTile = 32;
constexpr int kNT = 1024;          // threads of the single-CTA kernels
constexpr int kMaxSpecies = 16;
constexpr double kTol = 1.0e-8;    // distnorm convergence (slvfe.F90:1520)
constexpr int kItrMax = 100;
constexpr double kTiny = 1.0e-8;   // zero-bin tie (slvfe.F90:1180)

enum : int { kOk = 0, kErrNorm = 1, kErrExtrap = 2, kErrChol = 3, kErrZero = 4 };

thread_local const char* g_err = "";

// the first failing step's code stays: later kernels run on, as the host learns of it only at the end
__device__ void set_status(int* st, int code) { atomicCAS(st, 0, code); }

__device__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// fixed-order sum of one value per thread of a kNT-thread block
__device__ double block_sum(double v, double* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    double r = l < kNT / 32 ? sh[l] : 0.0;
    r = warp_sum(r);
    if (l == 0) sh[0] = r;
  }
  __syncthreads();
  return sh[0];
}

__device__ double block_max(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    double r = l < kNT / 32 ? sh[l] : -INFINITY;
    for (int o = 16; o > 0; o >>= 1) r = fmax(r, __shfl_down_sync(0xffffffffu, r, o));
    if (l == 0) sh[0] = r;
  }
  __syncthreads();
  return sh[0];
}

__device__ double block_min(double v, double* sh) { return -block_max(-v, sh); }

struct SlvArgs {
  int n, nsp;
  double kT;
  int n0;               // bins as read (before grouping)
  const double* rd0;    // rho in solution as read, for getslncv's threshold (slvfe.F90:884)
  const double* rr0;    // rho0 as read
  const double* rd;     // rho in solution as read (engstore-normalised)
  const double* rr;     // rho0 in the reference solvent as read
  const double* crd;    // bin coordinates (engsln's bin_middle)
  const int* spec;      // 1-based species of each bin
  double* rho;          // scaled rho
  double* rho0;         // scaled rho0
  double* nummol;       // [nsp] molecules per species
  double* omega;        // omega in solution
  int* both;            // 1: sampled in both systems
  double* harm;         // rho rho0 / (rho + rho0)
  double* reg;          // [nsp]
  int* status;
  const int* off;       // [nsp + 1] first bin of each species
  int functional;       // ERMOD_SLVFE_PYHNC / HNC / THNC / NONE
  double et;            // thnc threshold (kcal/mol)
};

// ---- distnorm's scaling and the directly sampled omega -------------------------------
__global__ void __launch_bounds__(kNT) k_slv_prep(SlvArgs a, double* __restrict__ corr) {
  __shared__ double sh[32];
  const int n = a.n;
  for (int p = 1; p <= a.nsp; ++p) {
    double s = 0.0, s0 = 0.0;
    for (int i = threadIdx.x; i < n; i += kNT)
      if (a.spec[i] == p) { s += a.rd[i]; s0 += a.rr[i]; }
    s = block_sum(s, sh);
    s0 = block_sum(s0, sh);
    const double nm = rint(s);
    if (threadIdx.x == 0) a.nummol[p - 1] = nm;
    const double f = s > 0.0 ? nm / s : 0.0, f0 = s0 > 0.0 ? nm / s0 : 0.0;
    for (int i = threadIdx.x; i < n; i += kNT)
      if (a.spec[i] == p) { a.rho[i] = a.rd[i] * f; a.rho0[i] = a.rr[i] * f0; }
  }
  __syncthreads();
  double mn = INFINITY, mn0 = INFINITY;
  for (int i = threadIdx.x; i < a.n0; i += kNT) {
    if (a.rd0[i] > 0.0) mn = fmin(mn, a.rd0[i]);
    if (a.rr0[i] > 0.0) mn0 = fmin(mn0, a.rr0[i]);
  }
  mn = block_min(mn, sh);
  mn0 = block_min(mn0, sh);
  for (int i = threadIdx.x; i < n; i += kNT) {
    const double r = a.rho[i], r0 = a.rho0[i];
    corr[i] = 1.0;
    const double rs = fmin(r / mn, 10.0), rr = fmin(r0 / mn0, 10.0);
    const int b = (rint(rs) >= 1.0 && rint(rr) >= 1.0) ? 1 : 0;
    a.both[i] = b;
    a.omega[i] = b ? -a.kT * log(r / r0) - a.crd[i] : 0.0;
    const double hs = r + r0;
    a.harm[i] = hs > 0.0 ? r * r0 / hs : 0.0;
  }
}

// ---- chmpot's grouping of consecutive bins (slvfe.F90:609-698) ------------------------
// merged bin k covers the bins [rng[k].x, rng[k].y) as read; rng[k].z = 1 for the last merged
// bin of a species, whose coordinate is that species' last coordinate as read
__global__ void k_slv_merge_vec(int g, const int4* __restrict__ rng, const double* __restrict__ rd,
                                const double* __restrict__ rr, const double* __restrict__ crd,
                                const int* __restrict__ spec, double* __restrict__ mrd, double* __restrict__ mrr,
                                double* __restrict__ mcrd, int* __restrict__ mspec) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= g) return;
  const int4 r = rng[k];
  double s = 0.0, s0 = 0.0, c = 0.0;
  for (int i = r.x; i < r.y; ++i) { s += rd[i]; s0 += rr[i]; c += crd[i]; }
  mrd[k] = s;
  mrr[k] = s0;
  mcrd[k] = r.z ? crd[r.y - 1] : c / (double)(r.y - r.x);
  mspec[k] = spec[r.x];
}

// column-major g x g sums of the n0 x n0 matrix over the bins of each merged pair, fixed order;
// element (i, j) of the input at j n0 + i, or at i n0 + j where it is row-major
__global__ void k_slv_merge_mat(int g, int n0, int row_major, const int4* __restrict__ rng,
                                const double* __restrict__ chi0, double* __restrict__ chi) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (size_t)g * g) return;
  const int r = (int)(e % g), c = (int)(e / g);
  const int4 R = rng[r], Cc = rng[c];
  double s = 0.0;
  for (int j = Cc.x; j < Cc.y; ++j)
    for (int i = R.x; i < R.y; ++i) s += chi0[row_major ? (size_t)i * n0 + j : (size_t)j * n0 + i];
  chi[e] = s;
}

// the unmerged matrix from row-major input: a transpose through shared memory, 32 x 32 a CTA
__global__ void k_slv_transpose(int n, const double* __restrict__ in, double* __restrict__ out) {
  __shared__ double t[kTile][kTile + 1];
  const int x0 = blockIdx.x * kTile, y0 = blockIdx.y * kTile, tx = threadIdx.x, ty = threadIdx.y;   // (32, 8)
  for (int j = ty; j < kTile; j += 8)
    if (y0 + j < n && x0 + tx < n) t[j][tx] = in[(size_t)(y0 + j) * n + x0 + tx];
  __syncthreads();
  for (int j = ty; j < kTile; j += 8)
    if (x0 + j < n && y0 + tx < n) out[(size_t)(x0 + j) * n + y0 + tx] = t[tx][j];
}

// ---- chi0 row scaling: one Gauss-Seidel sweep in three launches -----------------------
// Bin i's correction needs sum_j corr_j chi_ji with the bins j < i already updated.  k_slv_colsum
// forms the sums with the old corrections over the whole chip; k_slv_sweep then walks the bins 32
// at a time in one CTA: a warp updates the 32 in turn within their 32 x 32 block in shared memory
// while the others add the changes of the block before to the sums of the bins after.  The chain
// of quotients, one a bin, bounds it.  One CTA that formed
// every bin's sum in turn (a barrier pair and a column of the matrix a bin) took 2.98 ms a sweep
// at 1396 bins; the three launches take 0.52.
constexpr size_t kSumSmem = 160 * 1024;
constexpr int kCols = 8;      // 12 spill: 0.57 ms a sweep against 0.50

__global__ void __launch_bounds__(256) k_slv_colsum(SlvArgs a, const double* __restrict__ chi,
                                                    const double* __restrict__ corr, double* __restrict__ base) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, l = threadIdx.x & 31;
  if (i >= a.n) return;
  const double* col = chi + (size_t)i * a.n;
  for (int p = 0; p < a.nsp; ++p) {
    double v = 0.0;
    for (int j = a.off[p] + l; j < a.off[p + 1]; j += 32) v += corr[j] * col[j];
    v = warp_sum(v);
    if (l == 0) base[(size_t)p * a.n + i] = v;
  }
}

__global__ void __launch_bounds__(kNT) k_slv_sweep(SlvArgs a, const double* __restrict__ chi,
                                                   double* __restrict__ corr, double* __restrict__ gbase, int last,
                                                   int* __restrict__ done) {
  extern __shared__ double sbase[];            // the sums, where they fit (kSumSmem)
  __shared__ double T[kTile][kTile + 1], delta[2][kTile], sh[32];
  __shared__ double blk[kMaxSpecies][kTile];
  const int n = a.n, nsp = a.nsp, tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  double* base = gbase;
  if (sizeof(double) * (size_t)n * nsp <= kSumSmem) {
    base = sbase;
    for (int e = tid; e < n * nsp; e += kNT) base[e] = gbase[e];
    __syncthreads();
  }
  double err = 0.0;
  // row l, column w of a block, fetched a block ahead
  auto block_at = [&](int i0) {
    return i0 + l < n && i0 + w < n ? chi[(size_t)(i0 + w) * n + i0 + l] : 0.0;
  };
  // the sums of columns c, c + step, ... below end += the changes of the 32 bins from j0: a warp per
  // column, lanes over the rows, kCols columns in flight
  auto add_changes = [&](int j0, const double* dl, int c, int step, int end) {
    const int len = min(kTile, n - j0);
    const double d = l < len ? dl[l] : 0.0;
    int spl = 0, p0 = 0, p1 = 0;
    if (nsp > 1) {
      spl = a.spec[min(j0 + l, n - 1)] - 1;
      p0 = a.spec[j0] - 1;
      p1 = a.spec[j0 + len - 1] - 1;
    }
    for (; c < end; c += kCols * step) {
      double v[kCols];
#pragma unroll
      for (int u = 0; u < kCols; ++u)
        v[u] = c + u * step < end && l < len ? d * chi[(size_t)(c + u * step) * n + j0 + l] : 0.0;
      for (int p = p0; p <= p1; ++p) {                     // the block's species, almost always one
#pragma unroll
        for (int u = 0; u < kCols; ++u) {
          const double t = warp_sum(spl == p ? v[u] : 0.0);
          if (l == 0 && c + u * step < end) base[(size_t)p * n + c + u * step] += t;
        }
      }
    }
  };
  double next = block_at(0);
  int cur = 0;
  for (int i0 = 0; i0 < n; i0 += kTile, cur ^= 1) {
    const int len = min(kTile, n - i0);
    T[l][w] = next;
    next = block_at(i0 + kTile);
    if (w < nsp) blk[w][l] = l < len ? base[(size_t)w * n + i0 + l] : 0.0;
    __syncthreads();
    if (w == 0) {
      const bool on = l < len;
      const double old = on ? corr[i0 + l] : 0.0, r0 = on ? a.rho0[i0 + l] : 0.0;
      double mine = 0.0;
      if (nsp == 1) {
        // every lane keeps its sum's reciprocal y: a changed sum's is y (1 + t + t^2 + t^3) with
        // t = 1 - v y where the change is small (the rest below 1e-16), a quotient otherwise
        double v = blk[0][l], y = 1.0 / v;
        const double num = a.nummol[0];
        for (int j = 0; j < len; ++j) {
          const double now = v > 0.0 ? num * y * r0 : 0.0;     // final on lane j
          const double d = __shfl_sync(0xffffffffu, now - old, j);
          if (l == j) { mine = now; delta[cur][l] = d; }
          if (l > j) {
            v += d * T[j][l];
            const double t = fma(-v, y, 1.0);
            if (fabs(t) <= 1.0e-4) y = fma(y, fma(fma(t, t, t), t, t), y);
            else y = 1.0 / v;
          }
        }
      } else {
        const int sp = on ? a.spec[i0 + l] - 1 : 0;
        for (int j = 0; j < len; ++j) {
          double s = 0.0;
          for (int p = 0; p < nsp; ++p) {
            const double v = blk[p][l];
            if (v > 0.0) s += a.nummol[p] / v;
          }
          const double now = s / nsp * r0;
          const double d = __shfl_sync(0xffffffffu, now - old, j);
          const int pj = __shfl_sync(0xffffffffu, sp, j);
          if (l == j) { mine = now; delta[cur][l] = d; }
          if (l > j) blk[pj][l] += d * T[j][l];
        }
      }
      if (on) {
        corr[i0 + l] = mine;
        if (r0 > 0.0) err = fmax(err, fabs(mine - 1.0));
      }
    } else if (i0 > 0) {       // meanwhile the block before reaches the bins after this one
      add_changes(i0 - kTile, delta[cur ^ 1], i0 + kTile + w - 1, kNT / 32 - 1, n);
    }
    __syncthreads();
    add_changes(i0, delta[cur], i0 + kTile + w, kNT / 32, min(n, i0 + 2 * kTile));   // the next block at once
    __syncthreads();
  }
  err = block_max(err, sh);
  if (tid == 0) {
    *done = err <= kTol;
    if (!(err <= kTol) && last) set_status(a.status, kErrNorm);
  }
}

// chi *= corr corr^T
__global__ void k_slv_scale(int n, const double* __restrict__ corr, double* __restrict__ chi) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < (size_t)n * n) chi[e] *= corr[e % n] * corr[e / n];
}

// ---- omega in solution where one distribution is empty: weighted linear fit ----------
__global__ void k_slv_extrap(SlvArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = a.n;
  if (i >= n || a.both[i]) return;
  if (a.rho[i] <= 0.0) { a.omega[i] = 0.0; return; }
  const int sp = a.spec[i];
  auto same = [&](int k) { return a.spec[k] == sp && a.both[k]; };
  int m = 0, k = n - 1;
  for (int q = i - 1; q >= 0; --q) if (same(q)) { m = q; break; }
  for (int q = i + 1; q < n; ++q) if (same(q)) { k = q; break; }
  int j;
  if (a.both[m] && a.both[k]) j = abs(m - i) < abs(k - i) ? m : k;
  else if (a.both[m] || a.both[k]) j = a.both[m] ? m : k;
  else { set_status(a.status, kErrExtrap); return; }
  const double kT = a.kT, cj = a.crd[j], ci = a.crd[i];
  double wsum = 0.0;
  for (int q = 0; q < n; ++q) {
    if (!same(q)) continue;
    double sh = a.crd[q] - cj;
    if (q < i) sh = -sh - 2.0 * (cj - ci);
    const double wq = exp(-sh / kT) * a.harm[q];
    if (wq > 0.0) wsum += wq;
  }
  double m1 = 0.0, m2 = 0.0, my = 0.0, mxy = 0.0;
  for (int q = 0; q < n; ++q) {
    if (!same(q)) continue;
    double sh = a.crd[q] - cj;
    if (q < i) sh = -sh - 2.0 * (cj - ci);
    double wq = exp(-sh / kT) * a.harm[q];
    if (!(wq > 0.0)) continue;
    wq /= wsum;
    const double x = a.crd[q], y = a.omega[q];
    m1 += wq * x; m2 += wq * x * x; my += wq * y; mxy += wq * x * y;
  }
  const double den = m2 - m1 * m1;
  const double c0 = (m2 * my - m1 * mxy) / den, c1 = (mxy - m1 * my) / den;
  a.omega[i] = c0 + c1 * ci;
}

// ---- regularisation per species: trace of the sampled block / count^2 ----------------
__global__ void __launch_bounds__(kNT) k_slv_reg(SlvArgs a, const double* __restrict__ chi) {
  __shared__ double sh[32];
  const int n = a.n;
  for (int p = 1; p <= a.nsp; ++p) {
    double t = 0.0, c = 0.0;
    for (int i = threadIdx.x; i < n; i += kNT)
      if (a.spec[i] == p && a.rho0[i] > 0.0) {
        t += chi[(size_t)i * n + i] - a.rho0[i] * a.rho0[i];
        c += 1.0;
      }
    t = block_sum(t, sh);
    c = block_sum(c, sh);
    if (threadIdx.x == 0) a.reg[p - 1] = c > 0.0 ? t / (c * c) : 0.0;
  }
}

// ---- the padded system matrix and right-hand side ------------------------------------
__global__ void k_slv_build(SlvArgs a, const double* __restrict__ chi, int N, double* __restrict__ A,
                            double* __restrict__ A2, double* __restrict__ b, double* __restrict__ b2) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (size_t)N * N) return;
  const int r = (int)(e % N), c = (int)(e / N);   // column-major
  const int n = a.n;
  double v;
  if (r >= n || c >= n) {
    v = r == c ? 1.0 : 0.0;
  } else {
    const bool pr = a.rho0[r] > 0.0, pc = a.rho0[c] > 0.0;
    if (pr && pc) {
      v = chi[(size_t)c * n + r] - a.rho0[r] * a.rho0[c];
      if (a.spec[r] == a.spec[c]) v += a.reg[a.spec[r] - 1];
    } else {
      v = r == c ? 1.0 : 0.0;
    }
  }
  A[e] = v;
  A2[e] = v;
  if (c == 0) b[r] = b2[r] = (r < n && a.rho0[r] > 0.0) ? -a.kT * (a.rho[r] - a.rho0[r]) : 0.0;
}

// ---- blocked Cholesky, lower, column-major, 32 x 32 tiles ----------------------------
// Step k, one launch: a CTA per lower tile (i, j) of the trailing matrix forms its panel tiles
// P_i = A_ik L_kk^-T and P_j = A_jk L_kk^-T from the inverse of the diagonal factor (a product
// instead of a chain of 32 substitutions), and A_ij -= P_i P_j^T.  The CTAs of the first trailing
// column store P_i into L and carry the forward substitution, b_i -= P_i y_k with y_k = L_kk^-1 b_k;
// the first CTA factors and inverts its updated tile, the next step's diagonal, with one warp.  The
// steps form a serial chain (44 at 1396 bins), so a step's latency bounds the solve, not its
// arithmetic (0.9 GFLOP): 13 us a step, 7 of them the factor and inverse of one tile.  At 1396
// bins, factor and solve: 1.78 + 2.70 ms with a launch each for factor, panel and update and a
// solve whose tiles one thread substituted; 0.57 + 0.33 ms so.

// The factor's inverse of the symmetric tile t (lower part used) by warp 0: lane r holds row r of
// the tile and column r of the inverse; each column of the factor is passed on through `col`.
__device__ void chol_invert(const double (&t)[kTile][kTile + 2], double (&col)[kTile][kTile + 2],
                            double* __restrict__ inv, int* status) {
  const int r = threadIdx.x;
  double a[kTile], x[kTile];
#pragma unroll
  for (int c = 0; c < kTile; ++c) {
    a[c] = t[r][c];
    x[c] = c == r ? 1.0 : 0.0;
  }
#pragma unroll
  for (int j = 0; j < kTile; ++j) {
    const double d = __shfl_sync(0xffffffffu, a[j], j);
    if (r == j && !(d > 0.0)) set_status(status, kErrChol);
    const double ri = rsqrt(fmax(d, 1e-300));             // 1 / L_jj
    const double lj = a[j] * ri;
    col[j][r] = lj;
    x[j] *= ri;
    __syncwarp();
#pragma unroll
    for (int c = j + 1; c < kTile; ++c) {
      const double lc = col[j][c];
      a[c] -= lj * lc;
      x[c] -= lc * x[j];
    }
  }
#pragma unroll
  for (int i = 0; i < kTile; ++i) inv[i * kTile + r] = x[i];     // row i, column r
}

constexpr int kCholThreads = 256;

__global__ void __launch_bounds__(32) k_chol_first(const double* __restrict__ A, int N, double* __restrict__ Linv,
                                                   int* status) {
  __shared__ __align__(16) double t[kTile][kTile + 2], col[kTile][kTile + 2];
#pragma unroll 8
  for (int c = 0; c < kTile; ++c) t[threadIdx.x][c] = A[(size_t)c * N + threadIdx.x];
  __syncwarp();
  chol_invert(t, col, Linv, status);
}

__global__ void __launch_bounds__(kCholThreads) k_chol_step(double* __restrict__ A, int N, int kt,
    double* __restrict__ Lmat, double* __restrict__ Linv, double* __restrict__ b, double* __restrict__ y, int* status) {
  // rows of 34 doubles: 16-byte reads of consecutive rows fall in distinct banks
  __shared__ __align__(16) double V[kTile][kTile + 2], X[kTile][kTile + 2], Y[kTile][kTile + 2], P[kTile][kTile + 2],
      Q[kTile][kTile + 2], yk[kTile];
  // blockIdx.x enumerates the lower-triangle tile pairs (i, j), j <= i, of the trailing matrix
  int bl = blockIdx.x, j = 0;
  const int m = N / kTile - kt - 1;
  while (bl >= m - j) { bl -= m - j; ++j; }
  const int i = j + bl;
  const int r = threadIdx.x & 31, c0 = threadIdx.x >> 5;     // a thread takes columns c0 + 8 u of row r
  const int k0 = kt * kTile, i0 = (kt + 1 + i) * kTile, j0 = (kt + 1 + j) * kTile;
  double a[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int c = c0 + 8 * u;
    V[c][r] = Linv[(size_t)kt * kTile * kTile + c * kTile + r];          // row c, column r
    X[r][c] = A[(size_t)(k0 + c) * N + i0 + r];
    Y[r][c] = A[(size_t)(k0 + c) * N + j0 + r];
    a[u] = A[(size_t)(j0 + c) * N + i0 + r];
  }
  __syncthreads();
  double p[4] = {0.0, 0.0, 0.0, 0.0}, q[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
  for (int l = 0; l < kTile; l += 2) {
    const double2 xv = *(const double2*)&X[r][l], yv = *(const double2*)&Y[r][l];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double2 v = *(const double2*)&V[c0 + 8 * u][l];
      p[u] += xv.x * v.x; p[u] += xv.y * v.y;
      q[u] += yv.x * v.x; q[u] += yv.y * v.y;
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int c = c0 + 8 * u;
    P[r][c] = p[u];
    Q[r][c] = q[u];
    if (j == 0) Lmat[(size_t)(k0 + c) * N + i0 + r] = p[u];
  }
  if (j == 0 && c0 == 0) {
    double v = 0.0;
#pragma unroll 8
    for (int l = 0; l < kTile; ++l) v += V[r][l] * b[k0 + l];
    yk[r] = v;
    if (i == 0) y[k0 + r] = v;
  }
  __syncthreads();
  double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
  for (int l = 0; l < kTile; l += 2) {
    const double2 pv = *(const double2*)&P[r][l];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double2 qv = *(const double2*)&Q[c0 + 8 * u][l];
      v[u] += pv.x * qv.x; v[u] += pv.y * qv.y;
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int c = c0 + 8 * u;
    a[u] -= v[u];
    A[(size_t)(j0 + c) * N + i0 + r] = a[u];
    X[r][c] = a[u];
  }
  if (j == 0 && c0 == 7) {
    double v = 0.0;
#pragma unroll 8
    for (int l = 0; l < kTile; ++l) v += P[r][l] * yk[l];
    b[i0 + r] -= v;
  }
  if (i == 0 && j == 0) {
    __syncthreads();
    if (c0 == 0) chol_invert(X, V, Linv + (size_t)(kt + 1) * kTile * kTile, status);
  }
}

// L^T x = y, one CTA, tiles from the last: x_k = L_kk^-T y_k, then y_j -= L_kj^T x_k for the bins
// before.  y stays in shared memory; the next tile's inverse is fetched a tile ahead.
__global__ void __launch_bounds__(kNT) k_slv_back(const double* __restrict__ Lmat, const double* __restrict__ Linv,
                                                  int N, const double* __restrict__ b, const double* __restrict__ yg,
                                                  double* __restrict__ x) {
  extern __shared__ double y[];                // [N]
  __shared__ double xs[kTile], part[32][kTile + 1];
  const int nt = N / kTile, tid = threadIdx.x, w = tid >> 5, l = tid & 31;
  auto inv_at = [&](int kt) { return kt >= 0 ? Linv[(size_t)kt * kTile * kTile + w * kTile + l] : 0.0; };
  double next = inv_at(nt - 1);
  for (int e = tid; e < N - kTile; e += kNT) y[e] = yg[e];
  {   // the last tile's y, which no step formed
    const double v = warp_sum(next * b[(nt - 1) * kTile + l]);
    if (l == 0) y[(nt - 1) * kTile + w] = v;
  }
  __syncthreads();
  for (int kt = nt - 1; kt >= 0; --kt) {
    const int k0 = kt * kTile;
    // (L_kk^-T y)_c = sum_r V[r][c] y_r: warp w holds row w
    part[w][l] = next * y[k0 + w];
    next = inv_at(kt - 1);
    __syncthreads();
    {                                          // warp w adds column w
      const double v = warp_sum(part[l][w]);
      if (l == 0) {
        xs[w] = v;
        x[k0 + w] = v;
      }
    }
    __syncthreads();
    // a warp per column before the tile, lanes over its 32 rows, kCols columns in flight
    const double xl = xs[l];
    for (int c = w; c < k0; c += kCols * (kNT / 32)) {
      double v[kCols];
#pragma unroll
      for (int u = 0; u < kCols; ++u) {
        const int cu = c + u * (kNT / 32);
        v[u] = cu < k0 ? xl * Lmat[(size_t)cu * N + k0 + l] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < kCols; ++u) {
        const int cu = c + u * (kNT / 32);
        const double t = warp_sum(v[u]);
        if (l == 0 && cu < k0) y[cu] -= t;
      }
    }
    __syncthreads();
  }
}

// ---- posv_wrap's acceptance (slvfe.F90:520-531) against the regularised matrix Areg ----
// A CTA per 32 rows, the columns dealt to its warps (0.57 ms in one CTA, 0.013 so).  The maxima are of values >= 0, whose bit
// patterns order as integers; a NaN is passed over, as fmax does.
constexpr double kPosvResidual = 1.0e-6, kPosvAbs = 1.0e6;

__global__ void __launch_bounds__(kNT) k_slv_check(int n, int N, const double* __restrict__ Areg,
                                                   const double* __restrict__ rhs, const double* __restrict__ x,
                                                   unsigned long long* __restrict__ out) {
  __shared__ double part[32][33];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, r = blockIdx.x * 32 + l;
  double v = 0.0;
  if (r < n)
    for (int c = w; c < n; c += 32) v += Areg[(size_t)c * N + r] * x[c];
  part[w][l] = v;
  __syncthreads();
  if (w == 0 && r < n) {
    double s = 0.0;
    for (int q = 0; q < 32; ++q) s += part[q][l];
    atomicMax(out, (unsigned long long)__double_as_longlong(fmax(0.0, fabs(s - rhs[r]))));
    atomicMax(out + 1, (unsigned long long)__double_as_longlong(fmax(0.0, fabs(x[r]))));
  }
}

// ---- the eigen-decomposition fallback (getinscv, slvfe.F90:1124-1170) ------------------
// E = chi0 - rho0 rho0^T on the sampled bins, the identity elsewhere (n x n, column-major)
__global__ void k_slv_unreg(SlvArgs a, const double* __restrict__ chi, double* __restrict__ E) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int n = a.n;
  if (e >= (size_t)n * n) return;
  const int r = (int)(e % n), c = (int)(e / n);
  const bool pr = a.rho0[r] > 0.0, pc = a.rho0[c] > 0.0;
  E[e] = (pr && pc) ? chi[(size_t)c * n + r] - a.rho0[r] * a.rho0[c] : (r == c ? 1.0 : 0.0);
}

// coef[i] = (sum over sampled bins p of -kT (rho - rho0)_p V[p][i]) / lambda_i for i >= nsp
__global__ void k_slv_evd_coef(SlvArgs a, const double* __restrict__ V, const double* __restrict__ lam,
                               double* __restrict__ coef) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = a.n;
  if (i >= n) return;
  double s = 0.0;
  if (i >= a.nsp) {
    for (int p = 0; p < n; ++p)
      if (a.rho0[p] > 0.0) s += -a.kT * (a.rho[p] - a.rho0[p]) * V[(size_t)i * n + p];
    s /= lam[i];
  }
  coef[i] = s;
}

// x[p] = sum over i >= nsp of V[p][i] coef[i]
__global__ void k_slv_evd_x(SlvArgs a, const double* __restrict__ V, const double* __restrict__ coef,
                            double* __restrict__ x) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = a.n;
  if (p >= n) return;
  double s = 0.0;
  for (int i = a.nsp; i < n; ++i) s += V[(size_t)i * n + p] * coef[i];
  x[p] = s;
}

__device__ double pyhnc_soln(double f) { return f < 0.0 ? f + f / (exp(-f) - 1.0) + 1.0 : f / 2.0; }
__device__ double pyhnc_refs(double f) { return f < 0.0 ? log1p(-f) * (1.0 / f - 1.0) + 1.0 : f / 2.0; }

// chmpot's integrands (slvfe.F90:759-774): py-hnc, hnc / thnc (thnc, :1417-1436), none
__device__ void functional_terms(int functional, double om, double om0, double kT, double et, double* ls,
                                 double* lr) {
  switch (functional) {
    case ERMOD_SLVFE_HNC: *ls = om / kT / 2.0; *lr = om0 / kT / 2.0; return;
    case ERMOD_SLVFE_THNC: *ls = om / kT / 2.0; *lr = om0 < et ? 0.0 : om0 / kT / 2.0; return;
    case ERMOD_SLVFE_NONE: *ls = 0.0; *lr = 0.0; return;
    default: *ls = pyhnc_soln(om / kT); *lr = pyhnc_refs(om0 / kT); return;
  }
}

// ---- eczr zero shift, the functional and its per-species sums ------------------------
__global__ void __launch_bounds__(kNT) k_slv_chmpot(SlvArgs a, const double* __restrict__ x,
                                                    const double* __restrict__ aveuv, double* __restrict__ chmpt) {
  __shared__ double sh[32];
  __shared__ double zx[kMaxSpecies];
  const int n = a.n;
  __shared__ int pair[kMaxSpecies];     // upper bin of the species' last bin pair around zero energy
  if (threadIdx.x < a.nsp) pair[threadIdx.x] = -1;
  __syncthreads();
  for (int q = 1 + (int)threadIdx.x; q < n; q += kNT)
    if (a.spec[q] == a.spec[q - 1] && a.crd[q - 1] <= 0.0 && 0.0 <= a.crd[q]) atomicMax(&pair[a.spec[q] - 1], q);
  __syncthreads();
  if (threadIdx.x < a.nsp) {
    const int q = pair[threadIdx.x];
    int k = -1;
    if (q > 0) {
      const double lo = fabs(a.crd[q - 1]), hi = a.crd[q];
      if (hi > lo + kTiny) k = q - 1;
      else if (hi < lo - kTiny) k = q;
      else k = a.rho0[q - 1] >= a.rho0[q] ? q - 1 : q;
    }
    if (k < 0) set_status(a.status, kErrZero);
    zx[threadIdx.x] = k >= 0 ? x[k] : 0.0;
  }
  __syncthreads();
  const double kT = a.kT;
  for (int p = 1; p <= a.nsp; ++p) {
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += kNT) {
      if (a.spec[i] != p) continue;
      const double r = a.rho[i], r0 = a.rho0[i];
      if (!(r > 0.0 || r0 > 0.0)) continue;
      const double om0 = (r0 > 0.0 ? -kT * (r - r0) / r0 - x[i] : 0.0) + zx[p - 1];
      const double hs = r + r0;
      const double wt = r >= r0 ? 1.0 : 1.0 - ((r - r0) / (hs > 0.0 ? hs : 1.0)) * ((r - r0) / (hs > 0.0 ? hs : 1.0));
      double ls, lr;
      functional_terms(a.functional, a.omega[i], om0, kT, a.et, &ls, &lr);
      const double fac = wt * ls + (1.0 - wt) * lr;
      const double lcent = -(a.omega[i] + a.crd[i]);
      s += -kT * (r - r0) + lcent * r + kT * fac * (r - r0);
    }
    s = block_sum(s, sh);
    if (threadIdx.x == 0) chmpt[p - 1] = s + aveuv[p - 1];
  }
}

erm::WorkspaceCache g_ws;         // working memory and stream of a call

int fail(int code, const char* name) {
  g_err = name;
  return code;
}

template <class T>
cudaError_t dalloc(T** p, size_t n) { return cudaMalloc((void**)p, sizeof(T) * (n ? n : 1)); }

}  // namespace

extern "C" const char* ermod_slvfe_last_error(void) { return g_err; }

extern "C" void ermod_slvfe_release(void) { g_ws.release(); }

extern "C" int32_t ermod_slvfe_delta_mu(int32_t device, int32_t n0, int32_t nsp, int32_t group, int32_t inft,
                                        const double* rho_sln, const double* rho_ref, const double* chi_ref,
                                        const double* crd, const int32_t* spec, double kT, const double* aveuv,
                                        double slfeng, double* chmpt, double* total) {
  const ermod_slvfe_opts o{ERMOD_SLVFE_PYHNC, 1, 0.0};
  return ermod_slvfe_delta_mu_ex(device, n0, nsp, group, inft, rho_sln, rho_ref, chi_ref, crd, spec, kT, aveuv,
                                 slfeng, &o, chmpt, total, nullptr);
}

extern "C" int32_t ermod_slvfe_delta_mu_ex(int32_t device, int32_t n0, int32_t nsp, int32_t group, int32_t inft,
                                           const double* rho_sln, const double* rho_ref, const double* chi_ref,
                                           const double* crd, const int32_t* spec, double kT, const double* aveuv,
                                           double slfeng, const ermod_slvfe_opts* opts, double* chmpt,
                                           double* total, int32_t* used_evd) {
  return ermod_slvfe_delta_mu_layout(device, n0, nsp, group, inft, rho_sln, rho_ref, chi_ref, 0, crd, spec, kT, aveuv,
                                     slfeng, opts, chmpt, total, used_evd);
}

extern "C" int32_t ermod_slvfe_delta_mu_layout(int32_t device, int32_t n0, int32_t nsp, int32_t group, int32_t inft,
                                               const double* rho_sln, const double* rho_ref, const double* chi_ref,
                                               int32_t chi_row_major, const double* crd, const int32_t* spec,
                                               double kT, const double* aveuv, double slfeng,
                                               const ermod_slvfe_opts* opts, double* chmpt, double* total,
                                               int32_t* used_evd) {
  if (used_evd) *used_evd = 0;
  if (n0 < 2 || nsp < 1 || nsp > kMaxSpecies || group < 1 || inft < 0 || inft > 100 || !rho_sln || !rho_ref || !chi_ref || !crd || !spec ||
      !aveuv || !chmpt || !(kT > 0.0) || !opts || opts->functional < ERMOD_SLVFE_PYHNC ||
      opts->functional > ERMOD_SLVFE_NONE)
    return fail(ERMOD_ERR_ARG, "slv_arg");
  for (int i = 0; i < n0; ++i)
    if (spec[i] < 1 || spec[i] > nsp || (i > 0 && spec[i] < spec[i - 1])) return fail(ERMOD_ERR_ARG, "slv_arg");
  // chmpot's grouping (slvfe.F90:613-640): per species (bins - rduvcore * inft / 100) / group
  // merged bins, the last one taking the rest; rduvcore, the bins since the coordinate spacing
  // last stayed constant, counted as datread does (slvfe.F90:114-135).  The index bookkeeping
  // is host work, the sums run on the device.
  std::vector<int4> rng;
  std::vector<int> off(nsp + 1, 0);     // first merged bin of each species
  for (int i = 0; i < n0;) {
    int j = i;
    while (j < n0 && spec[j] == spec[i]) ++j;
    int core = 0;
    double dprev = 0.0;
    for (int q = i + 1; q < j; ++q) {
      const double d = crd[q] - crd[q - 1];
      if (q - i + 1 > 2) core = std::fabs(d - dprev) < 1.0e-8 ? 0 : core + 1;
      dprev = d;
    }
    const int m = (j - i - core * inft / 100) / group;
    if (m < 1) return fail(ERMOD_ERR_ARG, "slv_grp");
    for (int q = 0; q < m; ++q)
      rng.push_back(make_int4(i + q * group, q < m - 1 ? i + (q + 1) * group : j, q == m - 1 ? 1 : 0, 0));
    for (int p = spec[i]; p <= nsp; ++p) off[p] = (int)rng.size();
    i = j;
  }
  const int n = (int)rng.size();
  if (n < 2) return fail(ERMOD_ERR_ARG, "slv_grp");
  if ((size_t)n * sizeof(double) > 160 * 1024) return fail(ERMOD_ERR_ARG, "slv_siz");
  if (cudaSetDevice(device) != cudaSuccess) return fail(ERMOD_ERR_CUDA, "slv_cud");
  const int N = (n + kTile - 1) / kTile * kTile;
  const size_t nn = (size_t)n * n, NN = (size_t)N * N, nn0 = (size_t)n0 * n0;
  double *d_E = nullptr, *d_lam = nullptr, *d_coef = nullptr, *d_work = nullptr;
  int* d_info = nullptr;
  cusolverDnHandle_t sol = nullptr;
  int rc = ERMOD_OK;
  // one allocation for everything but the fallback's, in 256-byte steps
  size_t used = 0;
  auto take = [&](size_t bytes) {
    const size_t o = used;
    used += (bytes + 255) / 256 * 256;
    return o;
  };
  const size_t tiles = (size_t)(N / kTile);
  const size_t o_in = take(8 * (3 * (size_t)n0 + nsp)), o_spec0 = take(4 * (size_t)n0);
  const size_t o_rng = take(sizeof(int4) * (size_t)n), o_off = take(4 * (size_t)(nsp + 1)), o_chi0 = take(8 * nn0);
  const size_t o_rd = take(8 * (size_t)n), o_rr = take(8 * (size_t)n), o_crd = take(8 * (size_t)n);
  const size_t o_chi = group == 1 && inft == 0 && !chi_row_major ? o_chi0 : take(8 * nn);
  const size_t o_rho = take(8 * (size_t)n), o_rho0 = take(8 * (size_t)n), o_nm = take(8 * (size_t)nsp);
  const size_t o_om = take(8 * (size_t)n), o_harm = take(8 * (size_t)n), o_reg = take(8 * (size_t)nsp);
  const size_t o_corr = take(8 * (size_t)n), o_base = take(8 * (size_t)n * nsp);
  const size_t o_A = take(8 * NN), o_A2 = take(8 * NN), o_L = take(8 * NN), o_Li = take(8 * tiles * kTile * kTile);
  const size_t o_b = take(8 * (size_t)N), o_rhs = take(8 * (size_t)N), o_y = take(8 * (size_t)N), o_x = take(8 * (size_t)N);
  const size_t o_spec = take(4 * (size_t)n), o_both = take(4 * (size_t)n);
  // read back in one copy: the results, the check's two maxima, the status, the sweep's verdict
  const size_t o_out = take(8 * (size_t)(nsp + 2) + 8);
  erm::Workspace ws;
  bool ok = g_ws.take(device, used, ws);
  if (!ok) return fail(ERMOD_ERR_CUDA, "slv_mem");
  unsigned char* const arena = ws.p;
  const cudaStream_t st = ws.st;
  auto cleanup = [&]() {
    if (sol) cusolverDnDestroy(sol);
    for (void* p : {(void*)d_E, (void*)d_lam, (void*)d_coef, (void*)d_work, (void*)d_info})
      if (p) cudaFree(p);
    g_ws.give(ws, ok);
  };
  auto dp = [&](size_t o) { return (double*)(arena + o); };
  auto ip = [&](size_t o) { return (int*)(arena + o); };
  double *d_rd0 = dp(o_in), *d_rr0 = d_rd0 + n0, *d_crd0 = d_rr0 + n0, *d_av = d_crd0 + n0, *d_chi0 = dp(o_chi0);
  double *d_rd = dp(o_rd), *d_rr = dp(o_rr), *d_crd = dp(o_crd), *d_chi = dp(o_chi), *d_b = dp(o_x), *d_out = dp(o_out);
  double* d_chk = d_out + nsp;
  int *d_st = (int*)(d_chk + 2), *d_done = d_st + 1;
  std::vector<double> in(3 * (size_t)n0 + nsp);
  std::copy(rho_sln, rho_sln + n0, in.begin());
  std::copy(rho_ref, rho_ref + n0, in.begin() + n0);
  std::copy(crd, crd + n0, in.begin() + 2 * (size_t)n0);
  std::copy(aveuv, aveuv + nsp, in.begin() + 3 * (size_t)n0);
  ok = cudaMemcpyAsync(d_rd0, in.data(), 8 * in.size(), cudaMemcpyHostToDevice, st) == cudaSuccess;
  ok = ok && cudaMemcpyAsync(ip(o_spec0), spec, 4 * n0, cudaMemcpyHostToDevice, st) == cudaSuccess;
  ok = ok && cudaMemcpyAsync(arena + o_rng, rng.data(), sizeof(int4) * n, cudaMemcpyHostToDevice, st) == cudaSuccess;
  ok = ok && cudaMemcpyAsync(ip(o_off), off.data(), 4 * off.size(), cudaMemcpyHostToDevice, st) == cudaSuccess;
  ok = ok && cudaMemsetAsync(d_out, 0, 8 * (size_t)(nsp + 2) + 8, st) == cudaSuccess;
  ok = ok && erm::staged_to_device(d_chi0, chi_ref, 8 * nn0, st) == cudaSuccess;
  SlvArgs a{n, nsp, kT, n0, d_rd0, d_rr0, d_rd, d_rr, d_crd, ip(o_spec), dp(o_rho), dp(o_rho0), dp(o_nm), dp(o_om),
            ip(o_both), dp(o_harm), dp(o_reg), d_st, ip(o_off), opts->functional, opts->et};
  const int4* d_rng = (const int4*)(arena + o_rng);
  const size_t sum_smem = 8 * (size_t)n * nsp <= kSumSmem ? 8 * (size_t)n * nsp : 0;
  // per-device limits, set to the largest any call may ask for
  ok = ok && cudaFuncSetAttribute(k_slv_sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSumSmem) == cudaSuccess;
  ok = ok && cudaFuncSetAttribute(k_slv_back, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSumSmem + 256) == cudaSuccess;
  if (ok) {
    k_slv_merge_vec<<<(n + 127) / 128, 128, 0, st>>>(n, d_rng, d_rd0, d_rr0, d_crd0, ip(o_spec0), d_rd, d_rr, d_crd,
                                                     ip(o_spec));
    if (n == n0 && chi_row_major)
      k_slv_transpose<<<dim3((n + kTile - 1) / kTile, (n + kTile - 1) / kTile), dim3(kTile, 8), 0, st>>>(n, d_chi0, d_chi);
    else if (d_chi != d_chi0)
      k_slv_merge_mat<<<(unsigned)((nn + 255) / 256), 256, 0, st>>>(n, n0, chi_row_major, d_rng, d_chi0, d_chi);
    k_slv_prep<<<1, kNT, 0, st>>>(a, dp(o_corr));
    int done = 0;
    for (int it = 0; ok && !done && it < kItrMax; ++it) {
      k_slv_colsum<<<(n + 7) / 8, 256, 0, st>>>(a, d_chi, dp(o_corr), dp(o_base));
      k_slv_sweep<<<1, kNT, sum_smem, st>>>(a, d_chi, dp(o_corr), dp(o_base), it + 1 == kItrMax, d_done);
      k_slv_scale<<<(unsigned)((nn + 255) / 256), 256, 0, st>>>(n, dp(o_corr), d_chi);
      ok = cudaMemcpyAsync(&done, d_done, sizeof(int), cudaMemcpyDeviceToHost, st) == cudaSuccess &&
           cudaStreamSynchronize(st) == cudaSuccess;
    }
    k_slv_extrap<<<(n + 127) / 128, 128, 0, st>>>(a);
    k_slv_reg<<<1, kNT, 0, st>>>(a, d_chi);
    k_slv_build<<<(unsigned)((NN + 255) / 256), 256, 0, st>>>(a, d_chi, N, dp(o_A), dp(o_A2), dp(o_b), dp(o_rhs));
    k_chol_first<<<1, 32, 0, st>>>(dp(o_A), N, dp(o_Li), d_st);
    for (int kt = 0; kt + 1 < (int)tiles; ++kt) {
      const int m = (int)tiles - kt - 1;
      k_chol_step<<<m * (m + 1) / 2, kCholThreads, 0, st>>>(dp(o_A), N, kt, dp(o_L), dp(o_Li), dp(o_b), dp(o_y), d_st);
    }
    k_slv_back<<<1, kNT, 8 * (size_t)N, st>>>(dp(o_L), dp(o_Li), N, dp(o_b), dp(o_y), d_b);
    k_slv_check<<<(n + 31) / 32, kNT, 0, st>>>(n, N, dp(o_A2), dp(o_rhs), d_b, (unsigned long long*)d_chk);
    // the result on the Cholesky solution, read back with its verdict; run again if that is rejected
    k_slv_chmpot<<<1, kNT, 0, st>>>(a, d_b, d_av, d_out);
    ok = ok && cudaGetLastError() == cudaSuccess;
  }
  std::vector<double> got(nsp + 3);
  auto fetch = [&]() {
    return cudaMemcpyAsync(got.data(), d_out, 8 * got.size(), cudaMemcpyDeviceToHost, st) == cudaSuccess &&
           cudaStreamSynchronize(st) == cudaSuccess;
  };
  // posv_wrap's verdict decides between the Cholesky solution and the eigen-decomposition
  ok = ok && fetch();
  int status = 0;
  if (ok) std::memcpy(&status, &got[nsp + 2], sizeof(int));
  const double chk[2] = {got[nsp], got[nsp + 1]};
  const int first = status;             // a failure of the zero bin is only seen behind an accepted solution
  if (status == kErrZero) status = kOk;
  const bool rejected = status == kErrChol || (status == kOk && !(chk[0] <= kPosvResidual && chk[1] <= kPosvAbs));
  if (ok && rejected && opts->evd) {
    int lwork = 0, info = 0;
    ok = dalloc(&d_E, nn) == cudaSuccess && dalloc(&d_lam, n) == cudaSuccess && dalloc(&d_coef, n) == cudaSuccess &&
         dalloc(&d_info, 1) == cudaSuccess;
    ok = ok && cusolverDnCreate(&sol) == CUSOLVER_STATUS_SUCCESS && cusolverDnSetStream(sol, st) == CUSOLVER_STATUS_SUCCESS;
    if (ok) {
      k_slv_unreg<<<(unsigned)((nn + 255) / 256), 256, 0, st>>>(a, d_chi, d_E);
      ok = cudaGetLastError() == cudaSuccess;
    }
    ok = ok && cusolverDnDsyevd_bufferSize(sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, n, d_E, n, d_lam,
                                           &lwork) == CUSOLVER_STATUS_SUCCESS;
    ok = ok && dalloc(&d_work, (size_t)lwork) == cudaSuccess;
    ok = ok && cusolverDnDsyevd(sol, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, n, d_E, n, d_lam, d_work, lwork,
                                d_info) == CUSOLVER_STATUS_SUCCESS;
    ok = ok && cudaMemcpyAsync(&info, d_info, sizeof(int), cudaMemcpyDeviceToHost, st) == cudaSuccess;
    ok = ok && cudaStreamSynchronize(st) == cudaSuccess;
    if (ok && info != 0) status = kErrChol;   // "Failed inversion of correlation matrix" (slvfe.F90:1134)
    if (ok && info == 0) {
      k_slv_evd_coef<<<(n + 127) / 128, 128, 0, st>>>(a, d_E, d_lam, d_coef);
      k_slv_evd_x<<<(n + 127) / 128, 128, 0, st>>>(a, d_E, d_coef, d_b);
      ok = cudaGetLastError() == cudaSuccess;
      if (status == kErrChol) status = kOk;
      if (used_evd) *used_evd = 1;
    }
  } else if (ok && rejected && status == kOk) {
    status = kErrChol;   // the solution posv_wrap rejects, with the fallback switched off
  }
  if (ok && status == kOk && rejected) {
    ok = cudaMemsetAsync(d_st, 0, sizeof(int), st) == cudaSuccess;
    k_slv_chmpot<<<1, kNT, 0, st>>>(a, d_b, d_av, d_out);
    ok = ok && cudaGetLastError() == cudaSuccess && fetch();
    if (ok) std::memcpy(&status, &got[nsp + 2], sizeof(int));
  } else if (ok && status == kOk) {
    status = first;
  }
  if (ok) std::copy(got.begin(), got.begin() + nsp, chmpt);
  if (!ok) rc = fail(ERMOD_ERR_CUDA, "slv_cud");
  else if (status == kErrNorm) rc = fail(ERMOD_ERR_SLVFE, "slv_nrm");
  else if (status == kErrExtrap) rc = fail(ERMOD_ERR_SLVFE, "slv_ext");
  else if (status == kErrChol) rc = fail(ERMOD_ERR_SLVFE, "slv_chl");
  else if (status == kErrZero) rc = fail(ERMOD_ERR_SLVFE, "slv_zer");
  if (rc == ERMOD_OK && total) {
    double s = slfeng;
    for (int p = 0; p < nsp; ++p) s += chmpt[p];
    *total = s;
  }
  cleanup();
  return rc;
}
