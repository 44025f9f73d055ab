// pme_fused.cu -- the PME solve of a chunk of 32 targets without cuFFT and
// without a spread grid in HBM, for power-of-two meshes of 16..128 points a
// side.
//
// recpcal's per-insertion work (recpcal.F90:380-497 spreading, forward FFT,
// influence multiply, self energy; :592-710 the inverse FFT the gather reads)
// is, for a grid of K3 x K2 x K1 points and the half spectrum k1 < K1/2+1:
//
//   k_pme_plane     CTA = (target, k1 plane).  Forms the B-spline stencils of
//                   the solute sites (recpcal.F90:553-574) and their 1-D
//                   transforms B_m(k) = sum_c w_mc exp(-2 pi i k (g_m - c) / K_m)
//                   in FP64, builds the plane of the solute spectrum
//                   Qhat(k1, k2, k3) -- either directly,
//                   sum_a q_a B1_a(k1) B2_a(k2) B3_a(k3), or by spreading
//                   q_a B1_a(k1) w2 w3 on the (n2, n3) plane and a forward 2-D
//                   FFT -- multiplies by the influence function, adds the
//                   plane's share of the FP64 self energy, and runs the
//                   inverse 2-D FFT over (k2, k3) in shared memory.  The plane
//                   Y[b][k1][n3][n2] is written once (it stays in L2 for the
//                   next kernel).
//   k_pme_lines     a thread per (n3, n2) line and target: the complex-to-real
//                   transform along k1 (a half-length complex FFT of the
//                   Hermitian-packed line) in registers, written straight
//                   into the insertion-fastest potential layout the gather
//                   reads: n1 pairs (phi(2m), phi(2m+1)) per target, 32
//                   targets, for each line n3*K2 + n2
//                   (K1 <= 64; k_pme_lines128 does K1 = 128, k_pme_lines_few
//                   chunks of few targets).
//
// The FFTs are radix-8/4 Stockham stages (Govindaraju et al., "High
// performance discrete Fourier transforms on graphics processors", SC08):
// every thread holds its butterflies in registers across one barrier, so a
// stage runs in place in shared memory.  Twiddle tables are FP64 values
// rounded to FP32.  All sums run in a fixed order, so results are bitwise
// reproducible.  The result equals spreading + R2C + influence + C2R of the
// cuFFT path up to FP32 rounding.
#include <algorithm>
#include <cmath>

#include "engine.cuh"
#include "regfft.cuh"
#include "tc_sm100.cuh"

namespace erm {

using namespace fft;

namespace {

// Placement of a batch of 2^LNB transforms of length 2^LN in shared memory:
// transform bt starts at (bt >> LBG) * BPITCH + (bt & (2^LBG - 1)) * BSTRIDE
// and its elements are ES apart.  Everything is a compile-time constant, so
// shared-memory addresses are immediates off one register per butterfly.
template <int LN_, int LNB_, int LBG_, int BPITCH_, int BSTRIDE_, int ES_>
struct FftShape {
  static constexpr int LN = LN_, LNB = LNB_, LBG = LBG_, BPITCH = BPITCH_, BSTRIDE = BSTRIDE_, ES = ES_;
};

// One radix-R Stockham stage (input stride N/R, output groups of Ns = 2^LNS)
// of every transform of the batch, in place: each thread loads its
// butterflies, the block synchronises, then stores.  tw[m] = exp(-2 pi i m / N).
template <class S, int R, int LNS, int NTHR, bool INV>
__device__ __forceinline__ void fft_stage(float2* buf, const float2* __restrict__ tw, int tid) {
  constexpr int LR = R == 8 ? 3 : 2;
  constexpr int NR = 1 << (S::LN - LR), NS = 1 << LNS, LTS = S::LN - LNS - LR;
  constexpr int NBUT = (1 << (S::LN + S::LNB)) / R;
  constexpr int BPT = NBUT / NTHR;
  static_assert(BPT * NTHR == NBUT, "butterflies must divide evenly over the threads");
  float2 v[BPT][R];
  int dst[BPT];
#pragma unroll
  for (int i = 0; i < BPT; ++i) {
    const int idx = tid + i * NTHR;
    const int bt = idx & ((1 << S::LNB) - 1), j = idx >> S::LNB;
    const int off = (bt >> S::LBG) * S::BPITCH + (bt & ((1 << S::LBG) - 1)) * S::BSTRIDE;
    const int k = j & (NS - 1);
    const float2* src = buf + off + j * S::ES;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float2 x = src[r * NR * S::ES];
      if (LNS > 0 && r > 0) {                      // the first stage has k = 0: unit twiddles
        const float2 w = tw[(k * r) << LTS];
        x = INV ? make_float2(x.x * w.x + x.y * w.y, x.y * w.x - x.x * w.y) : cmul(x, w);
      }
      v[i][r] = x;
    }
    dft<R, INV>(v[i]);
    dst[i] = off + ((j - k) * R + k) * S::ES;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < BPT; ++i)
#pragma unroll
    for (int r = 0; r < R; ++r) buf[dst[i] + r * NS * S::ES] = v[i][r];
  __syncthreads();
}

// All stages of every transform of the batch: radix 8, radix 4 for the
// remaining factors (2^4 = 4 * 4 rather than 8 * 2; lengths are >= 8).
template <class S, int LNS, int NTHR, bool INV>
__device__ __forceinline__ void fft_stages(float2* buf, const float2* __restrict__ tw, int tid) {
  if constexpr (LNS < S::LN) {
    constexpr int REM = S::LN - LNS;
    constexpr int R = (REM >= 3 && REM != 4) ? 8 : 4;
    fft_stage<S, R, LNS, NTHR, INV>(buf, tw, tid);
    fft_stages<S, LNS + (R == 8 ? 3 : 2), NTHR, INV>(buf, tw, tid);
  }
}

template <class S, int NTHR, bool INV>
__device__ __forceinline__ void fft_batch(float2* buf, const float2* __restrict__ tw, int tid) {
  static_assert(S::LN >= 3, "transform length >= 8");
  fft_stages<S, 0, NTHR, INV>(buf, tw, tid);
}

constexpr int kSiteTile = 32;                  // solute sites staged in shared memory at a time (at most)
constexpr int kTabPairs = 8;                   // (target, site) pairs per CTA of k_site_tables
constexpr int kStn = 2 + 2 * kMaxOrder;        // stencil record: g2, g3, w2[kMaxOrder], w3[kMaxOrder]
constexpr int kLineRows = 4;                   // n2 rows per CTA of k_pme_lines (a warp each): 4 or 8
constexpr int kLoadBatch = 8;                  // global loads a thread keeps in flight while staging

template <int LK2, int LK3>
struct PlaneCfg {
  static constexpr int K2 = 1 << LK2, K3 = 1 << LK3, PITCH = K2 + 1;
  static constexpr int E = LK2 + LK3 <= 12 ? 16 : 32;     // plane points per thread
  static constexpr int NTHR = (K2 * K3) / E;
  static constexpr int MINB = E == 16 ? 3 : 1;
  // plane spreading accumulates in 2^-40 fixed point in shared memory when two
  // 64-bit sums a point fit (up to 8192 points)
  static constexpr bool FIXED = K2 * K3 <= 8192;
  static_assert(K3 % E == 0, "a thread owns E consecutive k3 of one k2 column");
};

}  // namespace

// ---------------------------------------------------------------------------
// k_site_tables: per (target, site) of a batch, the B-spline stencil
// (calc_spline_molecule, recpcal.F90:553-574) and its 1-D transforms
//   B_m(k) = sum_c w_mc exp(-2 pi i k (g_m - c) / K_m),
// summed in FP64 as exp(-2 pi i k g / K) times powers of exp(+2 pi i k / K).
// tab[pair][nk]: q B1(k1) for k1 < Kh1, then (direct sums) B2(k2), B3(k3).
// stn[pair][kStn]: g2, g3 (as floats), w2[kMaxOrder], w3[kMaxOrder].
// A CTA takes kTabPairs pairs: stencils first, then every entry of its pairs.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_site_tables(FrameArgs a, int base, int npairs, int nk,
    const float4* __restrict__ tgt_raw, const double2* __restrict__ fft_twd, float2* __restrict__ tab,
    float* __restrict__ stn) {
  __shared__ float sw[kTabPairs][3][kMaxOrder];
  __shared__ int sg[kTabPairs][3];
  __shared__ float sq[kTabPairs];
  const int K1 = a.K1, K2 = a.K2, K3 = a.K3, Kh1 = a.Kh1, n = a.order;
  const int p0 = blockIdx.x * kTabPairs;
  const int np = min(kTabPairs, npairs - p0);
  const float4* sites = tgt_raw + (size_t)base * a.nsite;
  for (int x = threadIdx.x; x < np * 3; x += blockDim.x) {
    const int t = x / 3, m = x - 3 * t;
    const float4 r = sites[p0 + t];
    const int K = m == 0 ? K1 : (m == 1 ? K2 : K3);
    float f = a.g.invcl[m][0] * r.x + a.g.invcl[m][1] * r.y + a.g.invcl[m][2] * r.z;
    f = f - floorf(f);
    f = f * (float)K;
    const int rci = (int)f;
    float w[kMaxOrder];
    spline_weights(f - (float)rci, n, w);
    for (int c = 0; c < kMaxOrder; ++c) sw[t][m][c] = c < n ? w[c] : 0.f;
    sg[t][m] = rci & (K - 1);
    if (m == 0) sq[t] = r.w;
  }
  __syncthreads();
  if (stn) {
    for (int x = threadIdx.x; x < np * kStn; x += blockDim.x) {
      const int t = x / kStn, r = x - t * kStn;
      float v;
      if (r < 2) v = (float)sg[t][1 + r];
      else if (r < 2 + kMaxOrder) v = sw[t][1][r - 2];
      else v = sw[t][2][r - 2 - kMaxOrder];
      stn[(size_t)(p0 + t) * kStn + r] = v;
    }
  }
  for (int x = threadIdx.x; x < np * nk; x += blockDim.x) {
    const int t = x / nk, r = x - t * nk;
    int m, k, K, t0;
    if (r < Kh1) { m = 0; k = r; K = K1; t0 = 0; }
    else if (r < Kh1 + K2) { m = 1; k = r - Kh1; K = K2; t0 = K1; }
    else { m = 2; k = r - Kh1 - K2; K = K3; t0 = K1 + K2; }
    const int g = sg[t][m];
    double2 e = fft_twd[t0 + ((k * g) & (K - 1))];
    const double2 st = fft_twd[t0 + ((K - k) & (K - 1))];   // exp(+2 pi i k / K)
    double re = (double)sw[t][m][0] * e.x, im = (double)sw[t][m][0] * e.y;
    for (int c = 1; c < n; ++c) {
      e = make_double2(e.x * st.x - e.y * st.y, e.x * st.y + e.y * st.x);
      re += (double)sw[t][m][c] * e.x;
      im += (double)sw[t][m][c] * e.y;
    }
    if (m == 0) {
      const double q = (double)sq[t];
      re *= q;
      im *= q;
    }
    tab[(size_t)(p0 + t) * nk + r] = make_float2((float)re, (float)im);
  }
}

// ---------------------------------------------------------------------------
// Direct site sums on the tensor cores (square 64 and 128 planes, up to 64 sites).  For one
// (target, k1) plane X(k3, k2) = sum_s B3_s(k3) D_s(k2), D_s = q_s B1_s(k1) B2_s(k2), is formed
// transposed, as one real product of a 128 x 2s operand A (row k2: Re D, Im D per site) by a
// 2s x 2K operand B (for each k3 the columns (Re B3, -Im B3) and (Im B3, Re B3)): product row
// k2, column 2 k3 + part is the real or imaginary part of X(k3, k2).  Every value is split
// into two TF32 terms (hi = v rounded to TF32, lo = v - hi rounded again) and the three
// products hi*hi, hi*lo and lo*hi are accumulated in FP32 in TMEM (`tcgen05.mma kind::tf32`,
// M = 128, N = 2K, K = 8 a step): the dropped lo*lo term and the split's rounding are below
// 2^-22 of each product, the FP32 level of the CUDA-core sums it replaces.  More than 16
// sites: tiles of 16 sites (K = 32) accumulate in the same TMEM columns, each tile's operands
// staged once the previous tile's MMAs have completed.
// ---------------------------------------------------------------------------
namespace tcs {
constexpr int kK = 32, kTileSites = kK / 2, kMaxSites = 4 * kTileSites;
constexpr int kRows = 128;                                          // M of every MMA
// A KN x KN plane, transposed: product row = k2 (KN = 64: rows 64..127 repeat rows 0..63, so
// that each of the four TMEM lane quarters holds the k2 of the warps that read it), product
// column = 2 k3 + part (part 0: Re, 1: Im), N = 2 KN.
template <int KN>
struct Shape {
  static_assert(KN == 64 || KN == 128, "64 x 64 or 128 x 128 planes");
  static constexpr int kN = 2 * KN;
  static constexpr int kAB = kRows * kK * 4;                      // bytes of the A operand (TF32)
  static constexpr int kBB = kN * kK * 4;                         // bytes of the B operand
  static constexpr int kOperandBytes = 2 * (kAB + kBB);           // hi and lo of each
  static constexpr int kTmemCols = kN;                            // 128 or 256
  static constexpr uint32_t kIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(kN >> 3) << 17) |
                                     ((uint32_t)(kRows >> 4) << 24);   // kind::tf32, D = F32, K-major
};

__device__ __forceinline__ uint32_t tf32_bits(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
// element (row, k) of a 128-byte-swizzled K-major tile, 32 TF32 a row
__device__ __forceinline__ uint32_t* slot(unsigned char* tile, int row, int k) {
  return (uint32_t*)(tile + tc::swz(row, k >> 2)) + (k & 3);
}
// The two TF32 terms of v.  The high one is rounded (to nearest, ties away from zero) by integer
// arithmetic: conversions run at a quarter of the rate and bounded the staging.  A NaN may lose its
// high term to the carry, but not the low one, v - hi.
struct Split {
  uint32_t hi, lo;
};
__device__ __forceinline__ Split split(float v) {
  const uint32_t h = (__float_as_uint(v) + 0x1000u) & 0xffffe000u;
  return {h, tf32_bits(v - __uint_as_float(h))};
}
__device__ __forceinline__ Split neg(Split v) { return {v.hi ^ 0x80000000u, v.lo ^ 0x80000000u}; }
// the pair (v0, v1) at columns (k, k + 1), k even: one 8-byte store into each of hi and lo
__device__ __forceinline__ void put2(unsigned char* hi, unsigned char* lo, int row, int k, Split v0, Split v1) {
  *reinterpret_cast<uint2*>(slot(hi, row, k)) = make_uint2(v0.hi, v1.hi);
  *reinterpret_cast<uint2*>(slot(lo, row, k)) = make_uint2(v0.lo, v1.lo);
}
__device__ __forceinline__ void put_split2(unsigned char* hi, unsigned char* lo, int row, int k, float v0, float v1) {
  put2(hi, lo, row, k, split(v0), split(v1));
}
// rows (2 c, 2 c + 1) of B: (Re, -Im) and (Im, Re)
__device__ __forceinline__ void put_b(unsigned char* hi, unsigned char* lo, int c, int k, float2 v) {
  const Split x = split(v.x), y = split(v.y);
  put2(hi, lo, 2 * c, k, x, neg(y));
  put2(hi, lo, 2 * c + 1, k, y, x);
}
__device__ __forceinline__ void mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  const uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      :
      : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(z), "r"(z), "r"(z), "r"(z));
}

// The product of k_pme_plane_pair (64 x 64 planes, two a CTA, 128 threads): staging, MMAs and bounded
// wait; returns the TMEM address of the product, which the caller reads and then frees with
// tmem_release.  Rows 0..63 of A hold D_s(k2) of plane k1A of the target whose site tables start at
// pairA, rows 64..127 those of plane k1B of the target at pairB (zero when k1B < 0).  Two targets take
// two rounds, each with its own B3 and the other half's A rows zero, accumulating in the same TMEM
// columns.  A CTA's staging is a chain of waits that nothing else hides (at most three CTAs an SM,
// in step): every table value of a tile is in flight at once, the next tile's during the products,
// and meanwhile() (the fetch of G) runs once the last tile is staged.
template <class F>
__device__ __forceinline__ uint32_t site_mma64(const float2* __restrict__ tab, size_t pairA, int k1A, size_t pairB,
                                               int k1B, int s, int nk, int Kh1, unsigned char* opnd, uint64_t* bar,
                                               uint32_t* tmem_slot, int* __restrict__ errflags, F meanwhile) {
  constexpr int KN = 64, NTHR = 128, NI = kTileSites * KN / NTHR;
  using Sh = Shape<KN>;
  using namespace tc;
  const int tid = threadIdx.x;
  // first: an SM starts its next CTA of such a kernel only once this one has given up the permit
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(Sh::kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  unsigned char* ahi = opnd;
  unsigned char* alo = ahi + Sh::kAB;
  unsigned char* bhi = alo + Sh::kAB;
  unsigned char* blo = bhi + Sh::kBB;
  // The item orders put the 16 lanes of a half warp on 16 distinct (16-byte chunk, half) slots of the
  // swizzled rows, so the 8-byte stores are free of bank conflicts: a lane's chunk is (t / 2) ^ (row
  // mod 8), its half t mod 2.
  // A item u: row k2 = qa, site ta + 2 u; B item u: rows of k3 = qb + 32 (u mod 2), site tb + 4 (u / 2)
  const int qa = (tid & 7) | (((tid >> 4) & 7) << 3), ta = (tid >> 3) & 1;
  const int qb = (tid & 3) | (((tid >> 4) & 7) << 2), tb = (tid >> 2) & 3;
  const bool cross = k1B >= 0 && pairB != pairA;
  const int tiles = (s + kTileSites - 1) / kTileSites, total = cross ? 2 * tiles : tiles;
  float2 cA[NI], cB[NI], b2[NI], b3[NI];
  auto load = [&](int tile) {                          // tile of a round: sites past s are zeros
    const bool second = tile >= tiles;
    const int t0 = (second ? tile - tiles : tile) * kTileSites;
    const bool onA = !second, onB = k1B >= 0 && (second || !cross);
    const float2* base = tab + (second ? pairB : pairA) * nk;
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      const int t = t0 + ta + 2 * u, v = t0 + tb + 4 * (u >> 1);
      cA[u] = cB[u] = b2[u] = b3[u] = make_float2(0.f, 0.f);
      if (t < s) {
        const float2* row = base + (size_t)t * nk;
        if (onA) cA[u] = __ldg(row + k1A);
        if (onB) cB[u] = __ldg(row + k1B);
        b2[u] = __ldg(row + Kh1 + qa);
      }
      if (v < s) b3[u] = __ldg(base + (size_t)v * nk + Kh1 + KN + qb + 32 * (u & 1));
    }
  };
  load(0);
  if (tid == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  bool ok = true;
  uint32_t tmem = 0;                                   // read once the first tile's barrier has passed (s >= 1)
  for (int tile = 0; tile < total && ok; ++tile) {
    const int ns = min(kTileSites, s - (tile >= tiles ? tile - tiles : tile) * kTileSites);
    // K steps of 8 columns that the tile's sites fill; the columns past 2 ns of the last step are zeros
    const int nks = (2 * ns + 7) / 8;
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      const int t = ta + 2 * u, v = tb + 4 * (u >> 1), k3 = qb + 32 * (u & 1);
      if (t < 4 * nks) {
        // q B1(k1) B2(k2 = qa); zero when off.  The roundings are fixed here, one form for each half (a
        // plane's last bits depend on its half), as earlier versions had them.
        const float2 d = make_float2(__fmaf_rn(cA[u].x, b2[u].x, -__fmul_rn(cA[u].y, b2[u].y)),
                                     __fmaf_rn(cA[u].y, b2[u].x, __fmul_rn(cA[u].x, b2[u].y)));
        put_split2(ahi, alo, qa, 2 * t, d.x, d.y);
        const float2 e = make_float2(__fmaf_rn(cB[u].x, b2[u].x, -__fmul_rn(cB[u].y, b2[u].y)),
                                     __fmaf_rn(cB[u].x, b2[u].y, __fmul_rn(cB[u].y, b2[u].x)));
        put_split2(ahi, alo, KN + qa, 2 * t, e.x, e.y);
      }
      if (v < 4 * nks) {
        put_b(bhi, blo, k3, 2 * v, b3[u]);
      }
    }
    if (tile + 1 < total) load(tile + 1);
    else meanwhile();
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = *tmem_slot;
    if (tid == 0) {
      const uint64_t dah = smem_desc(smem_u32(ahi)), dal = smem_desc(smem_u32(alo));
      const uint64_t dbh = smem_desc(smem_u32(bhi)), dbl = smem_desc(smem_u32(blo));
      for (int ks = 0; ks < nks; ++ks)
        mma(tmem, dah + 2 * ks, dbh + 2 * ks, Sh::kIdesc, (tile > 0 || ks > 0) ? 1u : 0u);
      for (int ks = 0; ks < nks; ++ks) mma(tmem, dah + 2 * ks, dbl + 2 * ks, Sh::kIdesc, 1u);
      for (int ks = 0; ks < nks; ++ks) mma(tmem, dal + 2 * ks, dbh + 2 * ks, Sh::kIdesc, 1u);
      mma_commit(bar);
    }
    // the tile's MMAs complete before its operands are overwritten or TMEM is read (bounded wait;
    // on expiry the error is flagged and the kernel waits once more, bounded, before going on)
    ok = __syncthreads_and(mbar_wait(bar, (uint32_t)(tile & 1))) != 0;
    if (!ok) {
      if (tid == 0) atomicOr(errflags, kErrTimeout);
      mbar_wait(bar, (uint32_t)(tile & 1));
    }
  }
  tc_fence_after();
  return tmem;
}

// every thread's TMEM reads are complete before warp 0 frees the columns
template <int KN>
__device__ __forceinline__ void tmem_release(uint32_t tmem) {
  tc::tc_fence_before();
  __syncthreads();
  if ((threadIdx.x >> 5) == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Shape<KN>::kTmemCols));
}

// The 128 x 128 plane's product: one target, one plane, tiles of 16 sites in two operand buffers
// (Shape<128>::kOperandBytes each), so that a tile is staged while the tensor cores work on the one
// before, from table values fetched a tile ahead.  The items are ordered as site_mma64's, free of bank
// conflicts (fetched a tile ahead, the shorter runs of table reads no longer cost what they save).
// Bars: two mbarriers.  Returns the TMEM address of the product; 512 threads.
__device__ __forceinline__ uint32_t site_mma128(const float2* __restrict__ tab, size_t pair0, int k1, int s, int nk,
                                                int Kh1, unsigned char* opnd, uint64_t* bar, uint32_t* tmem_slot,
                                                int* __restrict__ errflags) {
  constexpr int KN = 128, NTHR = 512, NI = kTileSites * KN / NTHR;
  using Sh = Shape<KN>;
  using namespace tc;
  const int tid = threadIdx.x;
  // A item u: x = tid + 512 u, q = x bits 0-2 and 4-7, site x bits 3 and 8-10
  // B item u: k3 = x bits 0-1 and 4-8, site x bits 2-3 and 9-10
  const int qa = (tid & 7) | (((tid >> 4) & 15) << 3), ta = ((tid >> 3) & 1) | ((tid >> 8) << 1);
  const int qb = (tid & 3) | (((tid >> 4) & 31) << 2), tb = (tid >> 2) & 3;
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(Sh::kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  float2 c1[NI], b2[NI], b3[NI];
  auto load = [&](int t0) {
#pragma unroll
    for (int u = 0; u < NI; ++u) {
      const int t = t0 + ta + 4 * u, v = t0 + tb + 4 * u;
      c1[u] = b2[u] = b3[u] = make_float2(0.f, 0.f);
      if (t < s) {
        const float2* row = tab + (pair0 + t) * nk;
        c1[u] = __ldg(row + k1);
        b2[u] = __ldg(row + Kh1 + qa);
      }
      if (v < s) b3[u] = __ldg(tab + (pair0 + v) * nk + Kh1 + KN + qb);
    }
  };
  load(0);
  bool ok = true;
  uint32_t tmem = 0;
  int tile = 0;
  for (int t0 = 0; t0 < s && ok; t0 += kTileSites, ++tile) {
    unsigned char* ahi = opnd + (tile & 1) * Sh::kOperandBytes;
    unsigned char* alo = ahi + Sh::kAB;
    unsigned char* bhi = alo + Sh::kAB;
    unsigned char* blo = bhi + Sh::kBB;
    if (tile >= 2) {   // the MMAs that read this buffer two tiles ago are done (bounded wait)
      ok = __syncthreads_and(mbar_wait(&bar[tile & 1], (uint32_t)((tile >> 1) - 1) & 1u)) != 0;
      if (!ok) break;
    }
    const int ns = min(kTileSites, s - t0), nks = (2 * ns + 7) / 8;
#pragma unroll
    for (int u = 0; u < NI; ++u) {   // sites past ns, up to the last K step's columns, are zeros
      const int t = ta + 4 * u, v = tb + 4 * u;
      if (t < 4 * nks) {
        const float2 d = fft::cmul(c1[u], b2[u]);             // q B1(k1) B2(k2 = qa)
        put_split2(ahi, alo, qa, 2 * t, d.x, d.y);
      }
      if (v < 4 * nks) {
        put_b(bhi, blo, qb, 2 * v, b3[u]);                    // B3(k3 = qb)
      }
    }
    load(t0 + kTileSites);
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    tmem = *tmem_slot;
    if (tid == 0) {
      const uint64_t dah = smem_desc(smem_u32(ahi)), dal = smem_desc(smem_u32(alo));
      const uint64_t dbh = smem_desc(smem_u32(bhi)), dbl = smem_desc(smem_u32(blo));
      for (int ks = 0; ks < nks; ++ks)
        mma(tmem, dah + 2 * ks, dbh + 2 * ks, Sh::kIdesc, (t0 > 0 || ks > 0) ? 1u : 0u);
      for (int ks = 0; ks < nks; ++ks) mma(tmem, dah + 2 * ks, dbl + 2 * ks, Sh::kIdesc, 1u);
      for (int ks = 0; ks < nks; ++ks) mma(tmem, dal + 2 * ks, dbh + 2 * ks, Sh::kIdesc, 1u);
      mma_commit(&bar[tile & 1]);
    }
  }
  // the last commit covers every MMA before it; on expiry of a wait the error is flagged and the kernel
  // waits once more, bounded, before going on
  const int last = tile - 1;
  if (ok) ok = __syncthreads_and(mbar_wait(&bar[last & 1], (uint32_t)(last >> 1) & 1u)) != 0;
  if (!ok) {
    if (tid == 0) atomicOr(errflags, kErrTimeout);
    const int w = tile > 0 ? tile - 1 : 0;
    mbar_wait(&bar[w & 1], (uint32_t)(w >> 1) & 1u);
    __syncthreads();
  }
  tc_fence_after();
  return tmem;
}
}  // namespace tcs

// ---------------------------------------------------------------------------
// k_pme_plane<LK2, LK3, DIRECT>: grid (k1max + 1, targets), K2*K3/E threads.  Thread
// tid owns the points (k2 = tid mod K2, k3 = (tid / K2) * E + e), e < E.
// Solute sites are staged ts at a time from the batch's site tables.
// ---------------------------------------------------------------------------
template <int LK2, int LK3, bool DIRECT>
__global__ void __launch_bounds__(PlaneCfg<LK2, LK3>::NTHR, PlaneCfg<LK2, LK3>::MINB) k_pme_plane(FrameArgs a,
    int tbase, int ts, const float2* __restrict__ tab, const float* __restrict__ stn,
    const float* __restrict__ engfacT, const float2* __restrict__ fft_tw, float2* __restrict__ Y,
    double* __restrict__ partial) {
  using C = PlaneCfg<LK2, LK3>;
  constexpr int K2 = C::K2, K3 = C::K3, PITCH = C::PITCH, E = C::E, NTHR = C::NTHR;
  extern __shared__ __align__(16) unsigned char psm[];
  const int k1 = blockIdx.x, b = blockIdx.y;
  const int K1 = a.K1, Kh1 = a.Kh1, s = a.nsite, n = a.order;
  const int nk = Kh1 + (DIRECT ? K2 + K3 : 0);
  const int tid = threadIdx.x;
  float2* tw2 = (float2*)psm;                          // [K2]
  float2* tw3 = tw2 + K2;                              // [K3]
  float2* plane = tw3 + K3;                            // [K3][PITCH]
  float2* c1 = plane + K3 * PITCH;                     // [ts] q_a B1_a(k1), padded to even length
  float2* b2 = c1 + ((ts + 1) & ~1);                   // DIRECT: [ts][K2] (16-byte aligned: K's are even)
  float2* b3 = b2 + (DIRECT ? ts * K2 : 0);            // DIRECT: [ts][K3]
  float* sst = (float*)b3;                             // spreading: [ts][kStn] stencils
  for (int p = tid; p < K2 + K3; p += NTHR) tw2[p] = fft_tw[K1 + p];
  const size_t pair0 = (size_t)(tbase + b) * s;       // first (target, site) pair of this target in the tables
  const int k2 = tid & (K2 - 1), k30 = (tid >> LK2) * E;
  float2 acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = make_float2(0.f, 0.f);
  if (!DIRECT && C::FIXED) {
    // q_a B1_a(k1) w2 w3 scattered on the (n2, n3) plane: a thread per (site, stencil point), in
    // 2^-40 fixed point (exact, order-independent), real and imaginary part in one pass.  Shared
    // memory has no 64-bit integer add, so a sum is two 32-bit words, the carry of the low one
    // added to the high one; rows of K2 + 4 put a site's 4 x 4 points on distinct banks.  Scaling by
    // 2^40 is exact in FP32, so one conversion rounds as the FP64 product did.
    // Measured with 200 sites on 64 x 64 planes, 32 targets x 27 planes: 77 ->
    // 43 us (one part at a time with 64-bit compare-and-swap adds and two divisions a point before).
    constexpr float kFix = 1099511627776.f;
    constexpr double kUnfix = 1.0 / 1099511627776.0;
    constexpr int FP = K2 + 4, NB = 4;
    uint32_t* facc = (uint32_t*)plane;                 // [re, im][low, high][K3][FP], under the plane
    for (int p = tid; p < K3 * FP; p += NTHR) ((uint4*)facc)[p] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    auto add = [&](uint32_t* at, float v) {
      const unsigned long long q = (unsigned long long)__float2ll_rn(v * kFix);
      const uint32_t lo = (uint32_t)q, old = atomicAdd(at, lo);
      atomicAdd(at + K3 * FP, (uint32_t)(q >> 32) + (old + lo < lo ? 1u : 0u));
    };
    const int nn = n * n, dt = NTHR / nn, dc = NTHR - dt * nn, inv = (65536 + n - 1) / n;
    int t = tid / nn, c = tid - t * nn;
    while (t < s) {
      float2 c1v[NB];
      float w2[NB], w3[NB];
      int at[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const size_t pair = pair0 + min(t, s - 1);
        const int c3 = (c * inv) >> 16, c2 = c - c3 * n;
        const float* st = stn + pair * kStn;
        c1v[u] = __ldg(tab + pair * nk + k1);
        const float2 g = __ldg((const float2*)st);
        w2[u] = __ldg(st + 2 + c2);
        w3[u] = __ldg(st + 2 + kMaxOrder + c3);
        at[u] = t < s ? (((int)g.y - c3) & (K3 - 1)) * FP + (((int)g.x - c2) & (K2 - 1)) : -1;
        t += dt;
        c += dc;
        if (c >= nn) {
          c -= nn;
          ++t;
        }
      }
#pragma unroll
      for (int u = 0; u < NB; ++u)
        if (at[u] >= 0) {
          add(facc + at[u], __fmul_rn(__fmul_rn(c1v[u].x, w2[u]), w3[u]));
          add(facc + 2 * K3 * FP + at[u], __fmul_rn(__fmul_rn(c1v[u].y, w2[u]), w3[u]));
        }
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const uint32_t* f = facc + (k30 + e) * FP + k2;
      const long long re = (long long)((unsigned long long)f[K3 * FP] << 32 | f[0]);
      const long long im = (long long)((unsigned long long)f[3 * K3 * FP] << 32 | f[2 * K3 * FP]);
      // most points are empty: no conversion
      acc[e].x = re ? (float)((double)re * kUnfix) : 0.f;
      acc[e].y = im ? (float)((double)im * kUnfix) : 0.f;
    }
    __syncthreads();
  } else {
    for (int a0 = 0; a0 < s; a0 += ts) {
      const int nt = min(ts, s - a0);
      __syncthreads();
      for (int x = tid; x < nt; x += NTHR) c1[x] = tab[(pair0 + a0 + x) * nk + k1];
      if (DIRECT) {
        // B2 then B3 of each site: K2 + K3 consecutive table entries, kLoadBatch loads in flight
        const int per = K2 + K3, tot = nt * per;
        for (int x0 = 0; x0 < tot; x0 += kLoadBatch * NTHR) {
          float2 v[kLoadBatch];
#pragma unroll
          for (int u = 0; u < kLoadBatch; ++u) {
            const int x = x0 + u * NTHR + tid;
            if (x < tot) v[u] = tab[(pair0 + a0 + x / per) * nk + Kh1 + x % per];
          }
#pragma unroll
          for (int u = 0; u < kLoadBatch; ++u) {
            const int x = x0 + u * NTHR + tid;
            if (x < tot) {
              const int t = x / per, r = x - t * per;
              if (r < K2) b2[t * K2 + r] = v[u];
              else b3[t * K3 + r - K2] = v[u];
            }
          }
        }
      } else {
        for (int x = tid; x < nt * kStn; x += NTHR) sst[x] = stn[(pair0 + a0) * kStn + x];
      }
      __syncthreads();
      if (DIRECT) {
        for (int t = 0; t < nt; ++t) {
          const float2 c = cmul(c1[t], b2[t * K2 + k2]);
          const float4* bt = (const float4*)(b3 + t * K3 + k30);   // two k3 per 16-byte load
#pragma unroll
          for (int e = 0; e < E; e += 2) {
            const float4 u = bt[e / 2];
            acc[e].x += c.x * u.x - c.y * u.y;
            acc[e].y += c.x * u.y + c.y * u.x;
            acc[e + 1].x += c.x * u.z - c.y * u.w;
            acc[e + 1].y += c.x * u.w + c.y * u.z;
          }
        }
      } else {
        // large planes: q_a B1_a(k1) w2 w3 accumulated in site order by the point's owner
        for (int t = 0; t < nt; ++t) {
          const float* st = sst + t * kStn;
          const int c2 = ((int)st[0] - k2) & (K2 - 1);
          if (c2 >= n) continue;
          const int g3 = (int)st[1];
          if (((g3 - k30) & (K3 - 1)) >= E + n - 1) continue;   // the site's rows miss this thread's rows
          const float2 c = c1[t];
          const float w2 = st[2 + c2];
          const float2 f = make_float2(c.x * w2, c.y * w2);
          const float* w3 = st + 2 + kMaxOrder;
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const int c3 = (g3 - (k30 + e)) & (K3 - 1);
            if (c3 < n) {
              acc[e].x += f.x * w3[c3];
              acc[e].y += f.y * w3[c3];
            }
          }
        }
      }
    }
  }
  // (DIRECT) acc holds Qhat(k1, k2, k3); otherwise the k1-transformed plane, still in (n2, n3)
  using Rows = FftShape<LK2, LK3, 30, 0, PITCH, 1>;
  using Cols = FftShape<LK3, LK2, 30, 0, 1, PITCH>;
  float2* own = plane + k30 * PITCH + k2;
  if (!DIRECT) {
#pragma unroll
    for (int e = 0; e < E; ++e) own[e * PITCH] = acc[e];
    __syncthreads();
    fft_batch<Rows, NTHR, false>(plane, tw2, tid);
    fft_batch<Cols, NTHR, false>(plane, tw3, tid);
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = own[e * PITCH];
  }
  // influence function and the plane's share of the self energy (recpcal.F90:482-497);
  // each mode's G |Qhat|^2 is formed in FP32 (~1e-7 relative) and summed in FP64
  double self = 0.0;
  const float* gk = engfacT + ((size_t)k1 * K3 + k30) * K2 + k2;
  float g[E];
#pragma unroll
  for (int e = 0; e < E; ++e) g[e] = gk[e * K2];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    self += (double)(g[e] * (acc[e].x * acc[e].x + acc[e].y * acc[e].y));
    own[e * PITCH] = make_float2(acc[e].x * g[e], acc[e].y * g[e]);
  }
  if (k1 == 0 || 2 * k1 == K1) self *= 0.5;
  __syncthreads();
  fft_batch<Rows, NTHR, true>(plane, tw2, tid);
  fft_batch<Cols, NTHR, true>(plane, tw3, tid);
  grid_dep_launch();                                  // the k1 transform may start filling the tail
  float2* y = Y + ((size_t)b * Kh1 + k1) * K3 * K2;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int p = tid + e * NTHR;
    y[p] = plane[(p >> LK2) * PITCH + (p & (K2 - 1))];
  }
  // the plane's share of the self energy, reduced in a fixed order; the k1 transform sums
  // the planes of each target (self_energy_sum)
  __shared__ double red[32];
  self = warp_sum(self);
  if ((tid & 31) == 0) red[tid >> 5] = self;
  __syncthreads();
  if (tid < 32) {
    double v = tid < (NTHR >> 5) ? red[tid] : 0.0;
    v = warp_sum(v);
    if (tid == 0) partial[(size_t)b * Kh1 + k1] = v;
  }
  // Launched behind the previous chunk's gather, which reads the potential grid that this
  // chunk's k1 transform overwrites: this grid does not complete before that gather has.
  grid_dep_wait();
}

// ---------------------------------------------------------------------------
// k_pme_plane_pair<LK>: two planes per CTA, K x K planes (K = 2^LK = 64), 2K threads.  The
// chunk's planes (target b, k1 <= k1max) are numbered p = b (k1max + 1) + k1 and a CTA takes
// p = 2c and 2c + 1 (c = plane_pair_of the CTA), so a chunk of 32 targets is at most
// 32 (k1max + 1) / 2 CTAs, one resident wave at 3 CTAs per SM for k1max < 27.  B3 does not
// depend on k1, so one tensor-core product serves two planes of a target: A rows 0..63 hold
// D(k2) of the first plane, rows 64..127 those of the second (zero past the chunk's last
// plane); a pair that spans two targets takes two rounds (tcs::site_mma64).  TMEM lane
// quarter w holds the rows that warp w reads.
// Thread (half = tid / K, k2 = tid mod K) takes all K of its column from TMEM, applies G,
// and transforms the column in registers (idft64_reg); a transpose through shared memory
// hands each thread a row n3 for the second axis, a second one the points of one n2, so that
// each warp store is one 256-byte row of Y.  Grid ceil(targets (k1max + 1) / 2).
// What bounds it is the chain of waits of a CTA, all in step.  Measured on 32 targets x 27
// planes: 24.8 -> 20.7 us with 12 sites, 37.0 -> 28.8 us with 32 (the ring's frame 3.23 -> 3.04
// ms) from the pairs of two targets placed first (they ended 4 us after the rest), tensor
// memory allocated first (an SM's CTAs start one after another, each when the one before has
// given up the permit: 3.2 -> 2.0 us for the three), the table values in flight together and
// fewer conversions in the staging.
// ---------------------------------------------------------------------------
// The pair that CTA c takes.  A pair that spans two targets (kp odd: one of kp in two targets) takes
// two rounds, so these pairs come first and do not make the launch's tail.
__device__ __forceinline__ int plane_pair_of(int c, int kp, int nb) {
  if ((kp & 1) == 0 || kp == 1) return c;
  const int spans = nb / 2;
  if (c < spans) return c * kp + (kp - 1) / 2;
  const int j = c - spans, m = j / (kp - 1), r = j - m * (kp - 1);
  return m * kp + r + (m < spans && r >= (kp - 1) / 2);
}
template <int LK>
__global__ void __launch_bounds__(2 << LK, 3) k_pme_plane_pair(FrameArgs a, int tbase, int nb,
    const float2* __restrict__ tab, const float* __restrict__ engfacT, Tw64 t64, float2* __restrict__ Y,
    double* __restrict__ partial, int* __restrict__ errflags) {
  constexpr int K = 1 << LK, NTHR = 2 * K, P = K + 1;
  static_assert(K == 64, "64 x 64 planes");
  extern __shared__ __align__(16) unsigned char psm[];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int half = tid >> LK, i = tid & (K - 1);          // plane of the pair; column k2, later row n3
  const int kp = a.k1max + 1, p0 = 2 * plane_pair_of(blockIdx.x, kp, nb);
  const bool has1 = p0 + 1 < nb * kp;
  const int b0 = p0 / kp, k1a = p0 - b0 * kp;
  const int b1 = has1 ? (p0 + 1) / kp : b0, k1b = has1 ? p0 + 1 - b1 * kp : -1;
  const bool live = half == 0 || has1;
  const int b = half ? b1 : b0, k1 = half && has1 ? k1b : k1a;
  const int Kh1 = a.Kh1, s = a.nsite, nk = Kh1 + 2 * K;
  unsigned char* opnd = (unsigned char*)(((uintptr_t)psm + 1023) & ~(uintptr_t)1023);
  float2* xp = (float2*)opnd + half * K * P;              // this plane's [n][P], over the dead operands
  float gv[K];                                            // G of column k2, fetched during the products
  __shared__ __align__(8) uint64_t tcs_bar;
  __shared__ uint32_t tcs_tmem;
  const uint32_t tmem =
      tcs::site_mma64(tab, (size_t)(tbase + b0) * s, k1a, (size_t)(tbase + b1) * s, k1b, s, nk, Kh1, opnd, &tcs_bar,
                      &tcs_tmem, errflags, [&]() {
                        const float* gk = engfacT + (size_t)k1 * K * K + i;
#pragma unroll
                        for (int e = 0; e < K; ++e) gv[e] = __ldg(gk + (size_t)e * K);
                      });
  // influence function and the plane's share of the self energy (recpcal.F90:482-497);
  // each mode's G |Qhat|^2 is formed in FP32 (~1e-7 relative) and summed in FP64
  float2 z[K];
  double part[4] = {0.0, 0.0, 0.0, 0.0};                  // four chains of FP64 adds
#pragma unroll
  for (int c = 0; c < 2 * K; c += 32) {
    uint32_t v[32];
    tc::tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int k3 = c / 2 + j;
      const float xr = __uint_as_float(v[2 * j]), xi = __uint_as_float(v[2 * j + 1]), g = gv[k3];
      part[j & 3] += (double)(g * __fmaf_rn(xr, xr, __fmul_rn(xi, xi)));
      z[k3] = make_float2(__fmul_rn(xr, g), __fmul_rn(xi, g));
    }
  }
  double self = (part[0] + part[1]) + (part[2] + part[3]);
  if (k1 == 0 || 2 * k1 == a.K1) self *= 0.5;
  tcs::tmem_release<K>(tmem);                             // also: every thread is past the MMAs
  // both axes run the same code, so that it is fetched once: column k2, then row n3
#pragma unroll 1
  for (int axis = 0; axis < 2; ++axis) {
    idft64_reg(z, t64);                                   // output n = 4 c + d at z[16 d + c]
    __syncthreads();
#pragma unroll
    for (int d = 0; d < 4; ++d)
#pragma unroll
      for (int c = 0; c < 16; ++c) xp[(4 * c + d) * P + i] = z[16 * d + c];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) z[k] = xp[i * P + k];     // after the columns: row n3 = i; after the rows: n2 = i
  }
  grid_dep_launch();                                      // the k1 transform may start filling the tail
  if (live) {
    float2* y = Y + ((size_t)b * Kh1 + k1) * K * K + i;
#pragma unroll
    for (int e = 0; e < K; ++e) y[(size_t)e * K] = z[e];
  }
  // each plane's share of the self energy over its two warps, in a fixed order; the k1
  // transform sums the planes of each target (self_energy_sum)
  __shared__ double red[NTHR / 32];
  self = warp_sum(self);
  if ((tid & 31) == 0) red[warp] = self;
  __syncthreads();
  if (i == 0 && live) partial[(size_t)b * Kh1 + k1] = red[2 * half] + red[2 * half + 1];
  // Launched behind the previous chunk's gather, which reads the potential grid that this
  // chunk's k1 transform overwrites: this grid does not complete before that gather has.
  grid_dep_wait();
}

// ---------------------------------------------------------------------------
// k_pme_plane128: one 128 x 128 plane a CTA of 512 threads, direct site sums on the tensor cores
// (site_mma128).  Each axis is the radix 8, 4, 4 transform of fft_stages with the same butterflies
// and twiddles, so the same roundings, but with the last two stages of a line's 16 points
// {k + 8 m} in one thread's registers: a line then crosses shared memory once between its first
// stage and the rest, not twice per stage.
//   thread (k2, q) takes k3 = 32 q .. of column k2 from TMEM, applies G and stores them;
//   rows (k2 -> n2): a warp owns eight rows k3; its exchange stays inside the row (position
//     9 (p / 8) + p mod 8 and rows of 152 points: free of bank conflicts);
//   columns (k3 -> n3): thread (n2, q) does the first-stage butterflies 4 q + i, exchanges through the
//     same array, finishes the points of k = 2 q, 2 q + 1 and stores them as 256-byte rows of Y.
// The plane crosses shared memory eight times where the stage by stage transform took fourteen.
// Measured on the 60-site chain, 2048 insertions into 32,768 waters (52 planes, four tiles of sites):
// the plane stage 21.5 -> 16.4 ms a frame, the frame 40.1 -> 35.1 ms.  With one CTA an SM (200 KB), its
// phases follow one another: issue slots 45 % busy, L1 and shared memory 49 %, tensor pipe 15 %.
// ---------------------------------------------------------------------------
constexpr int kRowPitch128 = 152;

// The last two radix-4 stages of a 128-point inverse transform for the 16 points p = k + 8 m (w[m]):
// on return w[4 r2 + r3] is output 8 r2 + k + 32 r3.  tw[m] = exp(-2 pi i m / 128).
__device__ __forceinline__ void idft128_tail(float2 (&w)[16], const float2 (&t2)[3], const float2 (&t3)[12]) {
  float2 o[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    float2 v[4] = {w[a], untwiddle(w[a + 4], t2[0]), untwiddle(w[a + 8], t2[1]), untwiddle(w[a + 12], t2[2])};
    dft<4, true>(v);
#pragma unroll
    for (int r = 0; r < 4; ++r) o[a][r] = v[r];
  }
#pragma unroll
  for (int r2 = 0; r2 < 4; ++r2) {
    float2 v[4] = {o[0][r2], untwiddle(o[1][r2], t3[3 * r2]), untwiddle(o[2][r2], t3[3 * r2 + 1]),
                   untwiddle(o[3][r2], t3[3 * r2 + 2])};
    dft<4, true>(v);
#pragma unroll
    for (int r = 0; r < 4; ++r) w[4 * r2 + r] = v[r];
  }
}
__device__ __forceinline__ void tail_twiddles(const float2* tw, int k, float2 (&t2)[3], float2 (&t3)[12]) {
#pragma unroll
  for (int r = 1; r < 4; ++r) {
    t2[r - 1] = tw[(k * r) << 2];
#pragma unroll
    for (int r2 = 0; r2 < 4; ++r2) t3[3 * r2 + r - 1] = tw[(8 * r2 + k) * r];
  }
}

__global__ void __launch_bounds__(512, 1) k_pme_plane128(FrameArgs a, int tbase, const float2* __restrict__ tab,
    const float* __restrict__ engfacT, const float2* __restrict__ fft_tw, float2* __restrict__ Y,
    double* __restrict__ partial, int* __restrict__ errflags) {
  constexpr int K = 128, RP = kRowPitch128;
  extern __shared__ __align__(16) unsigned char psm[];
  const int k1 = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int K1 = a.K1, Kh1 = a.Kh1, s = a.nsite, nk = Kh1 + 2 * K;
  float2* tw2 = (float2*)psm;                              // [K] of K2, then [K] of K3
  float2* tw3 = tw2 + K;
  unsigned char* opnd = (unsigned char*)(((uintptr_t)(tw3 + K) + 1023) & ~(uintptr_t)1023);
  float2* A = (float2*)opnd;                               // the plane, rows of RP points, over the dead operands
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ uint32_t tcs_tmem;
  for (int p = tid; p < 2 * K; p += 512) tw2[p] = fft_tw[K1 + p];
  const int col = (warp & 3) * 32 + lane, q = warp >> 2;   // TMEM lane quarter of this warp
  float g[32];                                             // G of this thread's points, fetched during the staging
  {
    const float* gk = engfacT + ((size_t)k1 * K + 32 * q) * K + col;
#pragma unroll
    for (int e = 0; e < 32; ++e) g[e] = __ldg(gk + (size_t)e * K);
  }
  const uint32_t tmem = tcs::site_mma128(tab, (size_t)(tbase + b) * s, k1, s, nk, Kh1, opnd, bars, &tcs_tmem, errflags);
  double self = 0.0;
  {
#pragma unroll
    for (int c = 0; c < 32; c += 8) {
      uint32_t x[2][8];
      const uint32_t t = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(2 * (32 * q + c));
      tc::tmem_ld8(t, x[0]);
      tc::tmem_ld8(t + 8, x[1]);
      tc::tmem_ld_wait();
      // influence function and the plane's share of the self energy (recpcal.F90:482-497);
      // each mode's G |Qhat|^2 is formed in FP32 (~1e-7 relative) and summed in FP64
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float xr = __uint_as_float(x[e >> 2][2 * (e & 3)]), xi = __uint_as_float(x[e >> 2][2 * (e & 3) + 1]);
        self += (double)(g[c + e] * (xr * xr + xi * xi));
        A[(32 * q + c + e) * RP + col] = make_float2(xr * g[c + e], xi * g[c + e]);
      }
    }
  }
  if (k1 == 0 || 2 * k1 == K1) self *= 0.5;
  tcs::tmem_release<K>(tmem);                              // also: the plane is in shared memory
  float2 v[4][8], w[2][16];
  {
    // rows k3 = 8 warp ..: first stage, lane (row parity, j)
    float2* R = A + (size_t)(8 * warp + (lane >> 4)) * RP;
    const int j = lane & 15;
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int r = 0; r < 8; ++r) v[t][r] = R[2 * t * RP + j + 16 * r];
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      dft<8, true>(v[t]);
#pragma unroll
      for (int r = 0; r < 8; ++r) R[2 * t * RP + 9 * j + r] = v[t][r];
    }
    __syncwarp();
  }
  {
    // the other two, lane (row, k)
    const int k = lane & 7;
    float2* R = A + (size_t)(8 * warp + (lane >> 3)) * RP + k;
    float2 t2[3], t3[12];
    tail_twiddles(tw2, k, t2, t3);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int m = 0; m < 16; ++m) w[h][m] = R[4 * h * RP + 9 * m];
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      idft128_tail(w[h], t2, t3);
#pragma unroll
      for (int r2 = 0; r2 < 4; ++r2)
#pragma unroll
        for (int r3 = 0; r3 < 4; ++r3) R[4 * h * RP + 8 * r2 + 32 * r3] = w[h][4 * r2 + r3];
    }
  }
  __syncthreads();
  // columns
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int r = 0; r < 8; ++r) v[i][r] = A[(4 * q + i + 16 * r) * RP + col];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    dft<8, true>(v[i]);
#pragma unroll
    for (int r = 0; r < 8; ++r) A[(8 * (4 * q + i) + r) * RP + col] = v[i][r];
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int m = 0; m < 16; ++m) w[h][m] = A[(2 * q + h + 8 * m) * RP + col];
  grid_dep_launch();                                       // the k1 transform may start filling the tail
  float2* y = Y + ((size_t)b * Kh1 + k1) * K * K + col;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float2 t2[3], t3[12];
    tail_twiddles(tw3, 2 * q + h, t2, t3);
    idft128_tail(w[h], t2, t3);
#pragma unroll
    for (int r2 = 0; r2 < 4; ++r2)
#pragma unroll
      for (int r3 = 0; r3 < 4; ++r3) y[(size_t)(8 * r2 + 2 * q + h + 32 * r3) * K] = w[h][4 * r2 + r3];
  }
  // the plane's share of the self energy, reduced in a fixed order; the k1 transform sums
  // the planes of each target (self_energy_sum)
  __shared__ double red[16];
  self = warp_sum(self);
  if (lane == 0) red[warp] = self;
  __syncthreads();
  if (warp == 0) {
    const double t = warp_sum(lane < 16 ? red[lane] : 0.0);
    if (lane == 0) partial[(size_t)b * Kh1 + k1] = t;
  }
  // Launched behind the previous chunk's gather, which reads the potential grid that this
  // chunk's k1 transform overwrites: this grid does not complete before that gather has.
  grid_dep_wait();
}

// selfrec[base + b] = sum over the planes k1 <= k1max of target b's shares, in
// plane order.  Run by the first CTA of the k1 transform: every plane of the
// chunk is complete by then.
__device__ __forceinline__ void self_energy_sum(const FrameArgs& a, int base, int nb, int Kh1,
                                                const double* __restrict__ partial, double* __restrict__ selfrec) {
  if (blockIdx.x != 0 || blockIdx.y != 0 || (int)threadIdx.x >= nb) return;
  const int b = threadIdx.x;
  double sum = 0.0;
  for (int k1 = 0; k1 <= a.k1max; ++k1) sum += partial[(size_t)b * Kh1 + k1];
  selfrec[base + b] = sum;
}

// ---------------------------------------------------------------------------
// k_pme_lines<LM>: the k1 transform into the potential grid for K1 = 2M <= 64, a thread per line.
// Grid (K3, K2 / kLineRows), 32 * kLineRows threads; warp j takes row
// n2 = blockIdx.y * kLineRows + j, lane b the target.  The CTA first stages
// the half spectra Y[b][k1][n3][n2], k1 <= k1max, of its kLineRows rows and
// 32 targets in shared memory (16-byte loads along n2), each line's k1 run
// contiguous: S[j JP + b LP + k1], LP = M + 2, JP = 32 LP + 4.  With these
// pitches a half warp's 8-byte staging stores and a quarter warp's 16-byte
// line reads fall on distinct banks, and a thread reads its line in M / 2 + 1
// 16-byte loads.  Each thread then packs its line (hermitian_pack), transforms
// it in registers (idft_reg) and writes the line's M pairs (phi(2n), phi(2n+1)):
// every store of a warp is one 256-byte row of the insertion-fastest layout.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int line_lp(int M) { return M + 2; }
__host__ __device__ constexpr int line_jp(int M) { return 32 * line_lp(M) + 4; }

size_t lines_smem(int M) { return sizeof(float2) * (size_t)kLineRows * line_jp(M); }

template <int LM>
__global__ void __launch_bounds__(32 * kLineRows, 2) k_pme_lines(FrameArgs a, int base, int nb,
    const float2* __restrict__ Y, Tw64 tw, const double* __restrict__ partial, double* __restrict__ selfrec,
    float* __restrict__ phi) {
  constexpr int M = 1 << LM, Kh1 = M + 1, NT = 32 * kLineRows;
  constexpr int LP = line_lp(M), JP = line_jp(M);
  static_assert(kLineRows == 4, "staging items: 2 row pairs x 2 k1 x 32 targets per 128 threads");
  extern __shared__ __align__(16) float2 S[];              // [kLineRows][32][LP] + pads
  const int K2 = a.K2, K3 = a.K3;
  const int tid = threadIdx.x;
  const int n3 = blockIdx.x, n2g = blockIdx.y * kLineRows;
  const size_t plane = (size_t)K3 * K2;
  const int kmax = a.k1max;
  grid_dep_wait();                                    // the planes of this chunk are complete
  self_energy_sum(a, base, nb, Kh1, partial, selfrec);
  {
    // staging item (u, x = tid): rows 2q, 2q + 1 of target bs at k1 = 2u + kp, one float4;
    // q = x mod 2, kp = bit 1, bs = bits 2-6, so a warp's loads are 16 whole 32-byte sectors
    const int q = tid & 1, kp = (tid >> 1) & 1, bs = ((tid >> 2) & 7) | (((tid >> 5) & 3) << 3);
    const bool on = bs < nb;
    const float4* src = (const float4*)(Y + (size_t)bs * Kh1 * plane + (size_t)n3 * K2 + n2g + 2 * q);
    float2* dst = S + (2 * q) * JP + bs * LP;
    // every load is issued before the first store, from a clamped (always valid) k1, so that
    // they are all in flight together; rows above k1max and targets past nb are not used
    constexpr int NPASS = (M + 2) / 2;                      // k1 = 0..M+1 in pairs
    static_assert(NT == 128, "one k1 pair per pass");
    float4 v[NPASS];
#pragma unroll
    for (int u = 0; u < NPASS; ++u) v[u] = __ldg(src + (size_t)min(2 * u + kp, kmax) * (plane / 2));
#pragma unroll
    for (int u = 0; u < NPASS; ++u) {
      const int k1 = 2 * u + kp;
      if (k1 <= kmax && k1 <= M) {
        const float4 t = on ? v[u] : make_float4(0.f, 0.f, 0.f, 0.f);
        dst[k1] = make_float2(t.x, t.y);
        dst[JP + k1] = make_float2(t.z, t.w);
      }
    }
  }
  __syncthreads();
  grid_dep_launch();                                  // the gather may start filling the tail
  const int b = tid & 31, j = tid >> 5;
  const float4* line = reinterpret_cast<const float4*>(S + j * JP + b * LP);
  float2 Z[M];
#pragma unroll
  for (int kk = 0; kk < M / 2; ++kk) {
    const float4 w = line[kk];
    Z[2 * kk] = 2 * kk <= kmax ? make_float2(w.x, w.y) : make_float2(0.f, 0.f);
    Z[2 * kk + 1] = 2 * kk + 1 <= kmax ? make_float2(w.z, w.w) : make_float2(0.f, 0.f);
  }
  float2 xM = make_float2(0.f, 0.f);
  if (M <= kmax) {
    const float4 w = line[M / 2];
    xM = make_float2(w.x, w.y);
  }
  hermitian_pack<LM>(Z, xM, tw);
  idft_reg<LM>(Z, tw);
  // z[n] = (phi(2n), phi(2n+1)): one 8-byte store per pair, a 256-byte row per warp
  float2* o = (float2*)phi + (size_t)(n3 * K2 + n2g + j) * M * kChunk + b;
#pragma unroll
  for (int n = 0; n < M; ++n) o[n * kChunk] = Z[n];
}

// ---------------------------------------------------------------------------
// k_pme_lines128: the same for K1 = 128, grid (K3, K2 / 16, targets / 8), 128 threads: 16 rows of n2
// of eight targets.  The half spectra of a chunk (218 MB on a 128^3 mesh) come from HBM, so what a CTA
// reads is cut for whole 128-byte lines: 16 consecutive n2 of one (target, k1), one 16-byte load a
// lane; it writes 64-byte runs (eight targets).  Shared layout: target b's row j at
// b (16 LP + 2) + j LP, LP = 66: a thread reads its line in 16-byte pieces free of bank conflicts.
// The 32-target, four-row CTAs with a staged shared-memory transform that this replaces read each line
// of Y in four 32-byte pieces from four CTAs: 60-site chain, 2048 insertions into 32,768 waters,
// the frame 35.1 -> 34.8 ms (16 targets of eight rows 36.1, 32 of four 38.3; the target groups are the
// fastest grid index, so that the 64-byte runs of a line of phi meet in L2: 36.8 with them slowest).
// ---------------------------------------------------------------------------
constexpr int kLines128Targets = 8, kLines128Rows = 128 / kLines128Targets;
constexpr int kLp128 = 66, kBp128 = kLines128Rows * kLp128 + 2;
size_t lines128_smem() { return sizeof(float2) * kLines128Targets * kBp128; }

__global__ void __launch_bounds__(128, 3) k_pme_lines128(FrameArgs a, int base, int nb, const float2* __restrict__ Y,
    const __grid_constant__ Tw128 tw, const double* __restrict__ partial, double* __restrict__ selfrec,
    float* __restrict__ phi) {
  constexpr int M = 64, Kh1 = M + 1, NB = 8;
  extern __shared__ __align__(16) float2 S[];
  const int K2 = a.K2, K3 = a.K3, tid = threadIdx.x, kmax = a.k1max;
  const int n3 = blockIdx.z, n2g = blockIdx.y * kLines128Rows, b0 = blockIdx.x * kLines128Targets;
  const size_t plane = (size_t)K3 * K2;
  grid_dep_wait();                                    // the planes of this chunk are complete
  if (n3 == 0) self_energy_sum(a, base, nb, Kh1, partial, selfrec);
  {
    // thread (row pair q, target b, k1 parity): rows 2 q, 2 q + 1 of k1 = kp, kp + 2, ...
    constexpr int NQ = kLines128Rows / 2;
    static_assert(NQ * kLines128Targets == 64, "two k1 a pass");
    const int q = tid % NQ, b = tid / NQ % kLines128Targets, kp = tid >> 6;
    const float4* src = (const float4*)(Y + (size_t)(b0 + b) * Kh1 * plane + (size_t)n3 * K2 + n2g + 2 * q);
    float2* dst = S + b * kBp128 + 2 * q * kLp128;
    // two k1 a pass; NB passes' loads in flight, from a clamped (always valid) k1
    for (int k0 = kp; k0 <= kmax; k0 += 2 * NB) {
      float4 v[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u) v[u] = __ldg(src + (size_t)min(k0 + 2 * u, kmax) * (plane / 2));
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        const int k1 = k0 + 2 * u;
        if (k1 <= kmax) {
          dst[k1] = make_float2(v[u].x, v[u].y);
          dst[kLp128 + k1] = make_float2(v[u].z, v[u].w);
        }
      }
    }
  }
  __syncthreads();
  grid_dep_launch();                                  // the gather may start filling the tail
  const int b = tid % kLines128Targets, j = tid / kLines128Targets;
  const float4* line = reinterpret_cast<const float4*>(S + b * kBp128 + j * kLp128);
  float2 Z[M];
#pragma unroll
  for (int kk = 0; kk < M / 2; ++kk) {
    const float4 w = line[kk];
    Z[2 * kk] = 2 * kk <= kmax ? make_float2(w.x, w.y) : make_float2(0.f, 0.f);
    Z[2 * kk + 1] = 2 * kk + 1 <= kmax ? make_float2(w.z, w.w) : make_float2(0.f, 0.f);
  }
  float2 xM = make_float2(0.f, 0.f);
  if (M <= kmax) {
    const float4 w = line[M / 2];
    xM = make_float2(w.x, w.y);
  }
  hermitian_pack<6>(Z, xM, tw);
  idft64_stages(Z, tw);
  float2* o = (float2*)phi + (size_t)(n3 * K2 + n2g + j) * M * kChunk + b0 + b;
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int r = 0; r < 8; ++r) o[(c + 8 * r) * kChunk] = Z[8 * c + r];
}

// ---------------------------------------------------------------------------
// k_pme_lines_few<LM>: the same transform for chunks of at most kFewTargets targets, a thread per
// (target, line), straight from Y (a warp's loads are a run of n2) into natural order,
// phi[b][line][n1].  The lane-a-target kernel above does 32 targets' lines whatever their number:
// one target on a 64^3 mesh took 13.7 us there, 4.5 here.
// ---------------------------------------------------------------------------
template <int LM>
__global__ void __launch_bounds__(128) k_pme_lines_few(FrameArgs a, int base, int nb, const float2* __restrict__ Y,
    Tw64 tw, const double* __restrict__ partial, double* __restrict__ selfrec, float* __restrict__ phi) {
  constexpr int M = 1 << LM, Kh1 = M + 1;
  const int plane = a.K3 * a.K2, line = blockIdx.x * 128 + threadIdx.x, b = blockIdx.y;
  const int kmax = a.k1max;
  grid_dep_wait();                                    // the planes of this chunk are complete
  self_energy_sum(a, base, nb, Kh1, partial, selfrec);
  grid_dep_launch();
  if (line >= plane) return;
  const float2* src = Y + (size_t)b * Kh1 * plane + line;
  float2 Z[M];
#pragma unroll
  for (int k = 0; k < M; ++k) Z[k] = k <= kmax ? __ldg(src + (size_t)k * plane) : make_float2(0.f, 0.f);
  const float2 xM = M <= kmax ? __ldg(src + (size_t)M * plane) : make_float2(0.f, 0.f);
  hermitian_pack<LM>(Z, xM, tw);
  idft_reg<LM>(Z, tw);
  float4* o = (float4*)(phi + ((size_t)b * plane + line) * (2 * M));
#pragma unroll
  for (int n = 0; n < M; n += 2) o[n / 2] = make_float4(Z[n].x, Z[n].y, Z[n + 1].x, Z[n + 1].y);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {
Tw64 make_tw64() {
  Tw64 t;
  for (int m = 0; m < 64; ++m) {
    const double ang = 2.0 * kPi * (double)m / 64.0;
    t.w[m] = make_float2((float)std::cos(ang), (float)-std::sin(ang));
  }
  return t;
}

Tw128 make_tw128() {
  Tw128 t;
  for (int m = 0; m < 128; ++m) {
    const double ang = 2.0 * kPi * (double)m / 128.0;
    t.w[m] = make_float2((float)std::cos(ang), (float)-std::sin(ang));
  }
  return t;
}

bool pow2_in(int k, int lo, int hi) { return k >= lo && k <= hi && (k & (k - 1)) == 0; }
int lg(int k) { int l = 0; while ((1 << l) < k) ++l; return l; }

int plane_elems(const FrameArgs& a) { return a.K2 * a.K3 <= 4096 ? 16 : 32; }

int site_tile(const FrameArgs& a) { return std::min(a.nsite, kSiteTile); }
int site_table_entries(const FrameArgs& a, bool direct) { return a.Kh1 + (direct ? a.K2 + a.K3 : 0); }

size_t plane_smem(const FrameArgs& a, bool direct) {
  const size_t ts = site_tile(a), tsa = (ts + 1) & ~(size_t)1;
  const size_t pts = (size_t)a.K2 * a.K3;
  const size_t tile = sizeof(float2) * tsa + (direct ? sizeof(float2) * ts * (a.K2 + a.K3)
                                                     : sizeof(float) * ts * kStn);
  const size_t tw = sizeof(float2) * (size_t)(a.K2 + a.K3), plane = sizeof(float2) * (size_t)a.K3 * (a.K2 + 1);
  // fixed-point spreading: two 64-bit sums a point, rows of K2 + 4, and the plane over them
  return tw + (!direct && pts <= 8192 ? 16 * (size_t)a.K3 * (a.K2 + 4) : plane + tile);
}

// k_pme_plane128: twiddles, then two operand buffers or the plane aliased over them, 1024-byte aligned
size_t plane_smem_128() {
  return sizeof(float2) * 256 + 1024 + std::max(sizeof(float2) * 128 * (size_t)kRowPitch128,
                                                2 * (size_t)tcs::Shape<128>::kOperandBytes);
}

// k_pme_plane_pair<LK>: the TF32 operands and, aliased over them, the two planes' K (K + 1)
// float2 rows, 1024-byte aligned
template <int LK>
size_t plane_smem_pair() {
  constexpr int K = 1 << LK;
  const size_t rows = sizeof(float2) * (size_t)(2 * K * (K + 1));
  return 1024 + std::max(rows, (size_t)tcs::Shape<K>::kOperandBytes);
}

// Compile-time plane sizes: every (K2, K3) in {16..128}^2 with K2 K3 >= 512.
#define ERM_PLANE_SIZES(X) \
  X(4, 5) X(4, 6) X(4, 7) X(5, 4) X(5, 5) X(5, 6) X(5, 7) X(6, 4) X(6, 5) X(6, 6) X(6, 7) X(7, 4) X(7, 5) X(7, 6) X(7, 7)

template <int L2, int L3>
cudaError_t plane_attr(const FrameArgs& a) {
  cudaError_t e = raise_smem_limit(k_pme_plane<L2, L3, true>, plane_smem(a, true));
  if (e == cudaSuccess) e = raise_smem_limit(k_pme_plane<L2, L3, false>, plane_smem(a, false));
  if constexpr (L2 == 7 && L3 == 7)
    if (e == cudaSuccess) e = raise_smem_limit(k_pme_plane128, plane_smem_128());
  if constexpr (L2 == 6 && L3 == 6)
    if (e == cudaSuccess) e = raise_smem_limit(k_pme_plane_pair<6>, plane_smem_pair<6>());
  return e;
}

template <int L2, int L3>
void plane_launch(const FrameArgs& a, const DeviceState& d, int tbase, int nb, bool direct, bool pdl, cudaStream_t s) {
  using C = PlaneCfg<L2, L3>;
  const dim3 grid(a.k1max + 1, nb);   // planes above k1max carry no influence-function weight
  const int ts = site_tile(a);
  int* err = d.status ? &d.status->flags : nullptr;
  if constexpr (L2 == 6 && L3 == 6) {
    if (direct && a.nsite <= tcs::kMaxSites) {   // site sums on the tensor cores, two planes per CTA
      static const Tw64 t64 = make_tw64();
      const int npairs = (nb * (a.k1max + 1) + 1) / 2;
      launch_k(pdl, dim3(npairs), 2 << L2, plane_smem_pair<6>(), s, k_pme_plane_pair<6>, a, tbase, nb,
               (const float2*)d.sitetab, (const float*)d.engfacT, t64, d.spec, d.partial, err);
      return;
    }
  }
  if constexpr (L2 == 7 && L3 == 7) {
    if (direct && a.nsite <= tcs::kMaxSites) {   // site sums on the tensor cores
      launch_k(pdl, grid, 512, plane_smem_128(), s, k_pme_plane128, a, tbase, (const float2*)d.sitetab,
               (const float*)d.engfacT, (const float2*)d.fft_tw, d.spec, d.partial, err);
      return;
    }
  }
  if (direct)
    launch_k(pdl, grid, C::NTHR, plane_smem(a, true), s, k_pme_plane<L2, L3, true>, a, tbase, ts,
             (const float2*)d.sitetab, (const float*)d.sitestn, (const float*)d.engfacT, (const float2*)d.fft_tw,
             d.spec, d.partial);
  else
    launch_k(pdl, grid, C::NTHR, plane_smem(a, false), s, k_pme_plane<L2, L3, false>, a, tbase, ts,
             (const float2*)d.sitetab, (const float*)d.sitestn, (const float*)d.engfacT, (const float2*)d.fft_tw,
             d.spec, d.partial);
}
}  // namespace

bool fused_supported(const FrameArgs& a) {
  if (!a.pme) return false;
  if (!pow2_in(a.K1, 16, 128) || !pow2_in(a.K2, 16, 128) || !pow2_in(a.K3, 16, 128)) return false;
  if (256 / (a.K1 / 2) > a.K2) return false;         // 16 x 16 planes at K1 = 16 stay on the cuFFT path
  if (a.K2 * a.K3 < 512) return false;               // at least 32 threads per plane
  if (a.K3 % plane_elems(a) != 0) return false;      // a thread owns E consecutive k3
  return plane_smem(a, true) <= 220 * 1024 && plane_smem(a, false) <= 220 * 1024;
}

int setup_fused(const FrameArgs& a) {
  if (!fused_supported(a)) return -1;
  const int l2 = lg(a.K2), l3 = lg(a.K3);
  cudaError_t e = cudaErrorInvalidValue;
#define ERM_ATTR(L2, L3) if (l2 == L2 && l3 == L3) e = plane_attr<L2, L3>(a);
  ERM_PLANE_SIZES(ERM_ATTR)
#undef ERM_ATTR
  if (e != cudaSuccess) return -1;
  const int lm = lg(a.K1 / 2);
  if (lm == 3) e = raise_smem_limit(k_pme_lines<3>, lines_smem(8));
  if (lm == 4) e = raise_smem_limit(k_pme_lines<4>, lines_smem(16));
  if (lm == 5) e = raise_smem_limit(k_pme_lines<5>, lines_smem(32));
  if (lm == 6) e = raise_smem_limit(k_pme_lines128, lines128_smem());
  return e == cudaSuccess ? 0 : -1;
}

size_t fused_sitetab_elems(const FrameArgs& a, int batch, bool direct) {
  return (size_t)batch * a.nsite * site_table_entries(a, direct);
}
size_t fused_sitestn_elems(const FrameArgs& a, int batch) { return (size_t)batch * a.nsite * kStn; }

void fused_twiddles(int K1, int K2, int K3, std::vector<float2>& tw, std::vector<double2>& twd) {
  // [K1 | K2 | K3] tables of exp(-2 pi i m / N), FP64 rounded to FP32 and in FP64
  tw.clear();
  twd.clear();
  const int Ns[3] = {K1, K2, K3};
  for (int t = 0; t < 3; ++t)
    for (int m = 0; m < Ns[t]; ++m) {
      const double ang = 2.0 * kPi * (double)m / (double)Ns[t];
      const double c = std::cos(ang), sn = -std::sin(ang);
      tw.push_back(make_float2((float)c, (float)sn));
      twd.push_back(make_double2(c, sn));
    }
}

void launch_site_tables(const FrameArgs& a, const DeviceState& d, int bb, int nbatch, bool direct, cudaStream_t s) {
  const int npairs = nbatch * a.nsite;
  k_site_tables<<<(npairs + kTabPairs - 1) / kTabPairs, 256, 0, s>>>(a, bb, npairs, site_table_entries(a, direct),
                                                                     d.tgt_raw, d.fft_twd, d.sitetab,
                                                                     direct ? nullptr : d.sitestn);
}

void launch_pme_plane(const FrameArgs& a, const DeviceState& d, int tbase, int nb, bool direct, bool pdl,
                      cudaStream_t s) {
  const int l2 = lg(a.K2), l3 = lg(a.K3);
#define ERM_LAUNCH(L2, L3) if (l2 == L2 && l3 == L3) plane_launch<L2, L3>(a, d, tbase, nb, direct, pdl, s);
  ERM_PLANE_SIZES(ERM_LAUNCH)
#undef ERM_LAUNCH
}

void launch_pme_rows(const FrameArgs& a, const DeviceState& d, int base, int nb, bool pdl, cudaStream_t s) {
  static const Tw64 tw = make_tw64();
  const dim3 lgrid(a.K3, a.K2 / kLineRows);
  if (few_targets(a, d, nb)) {
    const dim3 fgrid((a.K3 * a.K2 + 127) / 128, nb);
#define ERM_FEW(LM) launch_k(pdl, fgrid, 128, 0, s, k_pme_lines_few<LM>, a, base, nb, (const float2*)d.spec, tw, \
      (const double*)d.partial, d.selfrec, d.phi)
    if (a.K1 == 16) ERM_FEW(3);
    else if (a.K1 == 32) ERM_FEW(4);
    else ERM_FEW(5);
#undef ERM_FEW
    return;
  }
  switch (lg(a.K1 / 2)) {
    case 3:
      launch_k(pdl, lgrid, 32 * kLineRows, lines_smem(1 << 3), s, k_pme_lines<3>, a, base, nb, (const float2*)d.spec,
               tw, (const double*)d.partial, d.selfrec, d.phi);
      return;
    case 4:
      launch_k(pdl, lgrid, 32 * kLineRows, lines_smem(1 << 4), s, k_pme_lines<4>, a, base, nb, (const float2*)d.spec,
               tw, (const double*)d.partial, d.selfrec, d.phi);
      return;
    case 5:
      launch_k(pdl, lgrid, 32 * kLineRows, lines_smem(1 << 5), s, k_pme_lines<5>, a, base, nb, (const float2*)d.spec,
               tw, (const double*)d.partial, d.selfrec, d.phi);
      return;
    default: break;
  }
  static const Tw128 t128 = make_tw128();
  launch_k(pdl, dim3((nb + kLines128Targets - 1) / kLines128Targets, a.K2 / kLines128Rows, a.K3), 128, lines128_smem(), s,
           k_pme_lines128, a, base, nb, (const float2*)d.spec, t128, (const double*)d.partial, d.selfrec, d.phi);
}

}  // namespace erm
