// mlp.cu -- the learned insertion proposal's network: a 64-128-128-128-1
// multilayer perceptron over a voxel's 4x4x4 local solvent-density grid,
// BF16 weights with FP32 accumulation, trained on the device by the kernels
// below (no library GEMM, no autograd).  No reference counterpart: erdst
// inserts uniformly (insertion.F90:152-162); the proposal only changes where
// insertions go and carries the importance weight p/q that keeps every
// histogram and ecorr increment unbiased.
//
//   forward   h1 = relu(W1 x + b1), h2 = relu(W2 h1 + b2), h3 = relu(W3 h2 + b3),
//             s = w4 . h3 + b4                      (the voxel's logit)
//   loss      mean binary cross-entropy with logits, softplus(s) - y s
//   backward  the chain rule through the same BF16 weights; every gradient
//             element is one thread's fixed-order sum over the batch, so the
//             gradients are bitwise reproducible
//   update    Adam on FP32 master weights, rounded to BF16 for the next pass
//
// Parameter vector layout (FP32, ERMOD_MLP_NPARAMS entries):
//   W1[128][64] b1[128] W2[128][128] b2[128] W3[128][128] b3[128] w4[128] b4
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "engine.cuh"
#include "tc_sm100.cuh"

namespace erm {

namespace {

// ---- the backward pass -------------------------------------------------------
// One CTA per kBwdRows samples runs the whole chain of its rows in shared memory: the loss and
// dL/ds, d3 = gs w4^T [h3 > 0], d2 = (d3 W3) [h2 > 0], d1 = (d2 W2) [h1 > 0], and its rows' share
// of every gradient, written as one row of `part` in the parameter layout; k_bwd_sum adds the
// rows of `part` in order.  Every gradient element is a fixed-order FP32 sum: over the rows of a
// CTA, then over the CTAs, so gradients are bitwise reproducible.
//
// The layer-by-layer products this replaces ran the three weight gradients (128 x 128 sums over
// the batch) on four CTAs each, a serial chain over the 4096 samples: 2.22 ms of a 2.6 ms call,
// and the bias sums 0.30 ms on one warp each.  Split over the samples, 128 CTAs fill the chip once
// and the intermediates d1..d3 stay in shared memory: k_bwd 34 us, k_bwd_sum 7 us, the call 213 us.
// The products are FP32 FMAs (0.74 GFLOP a batch of 4096, about 10 us of the chip's FMA pipes), one
// CTA an SM by its 168 KB; what is left is the staging and the shared-memory reads of the products.
// The partial rows (21 MB) stay in L2.
constexpr int kBwdRows = 32, kBwdThreads = 256;
constexpr int kBwdParts = 296;     // rows of `part` at most (two waves of one CTA an SM): larger batches loop
__host__ __device__ inline int bwd_parts(int n) {
  const int nt = (n + kBwdRows - 1) / kBwdRows;
  return nt < kBwdParts ? nt : kBwdParts;
}

struct BwdSmem {
  float h3[kBwdRows][kMlpHidden], h2[kBwdRows][kMlpHidden], h1[kBwdRows][kMlpHidden], x[kBwdRows][kMlpIn];
  float d3[kBwdRows][kMlpHidden], d2[kBwdRows][kMlpHidden], d1[kBwdRows][kMlpHidden];
  __nv_bfloat16 w3[kMlpHidden * kMlpHidden], w2[kMlpHidden * kMlpHidden];
  float gs[kBwdRows];
};
static_assert(sizeof(BwdSmem) <= 227 * 1024, "one CTA's rows and both weight matrices in shared memory");

// out[r][k] = [h[r][k] > 0] sum_j d[r][j] W[j][k], j in order: warp w takes rows 4w..4w+3, a lane four columns
__device__ __forceinline__ void bwd_layer(const float (&d)[kBwdRows][kMlpHidden], const __nv_bfloat16* w,
                                          const float (&h)[kBwdRows][kMlpHidden], float (&out)[kBwdRows][kMlpHidden]) {
  const int r0 = (threadIdx.x >> 5) * 4, k0 = (threadIdx.x & 31) * 4;
  float acc[4][4] = {};
#pragma unroll 2
  for (int j0 = 0; j0 < kMlpHidden; j0 += 4) {
    float4 dv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) dv[i] = *(const float4*)&d[r0 + i][j0];
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      const uint2 wp = *(const uint2*)(w + (j0 + jj) * kMlpHidden + k0);
      // a BF16 is the high half of its FP32 pattern
      const float wv[4] = {__uint_as_float(wp.x << 16), __uint_as_float(wp.x & 0xffff0000u),
                           __uint_as_float(wp.y << 16), __uint_as_float(wp.y & 0xffff0000u)};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float dd = jj == 0 ? dv[i].x : jj == 1 ? dv[i].y : jj == 2 ? dv[i].z : dv[i].w;
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[i][k] = fmaf(dd, wv[k], acc[i][k]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < 4; ++k) out[r0 + i][k0 + k] = h[r0 + i][k0 + k] > 0.f ? acc[i][k] : 0.f;
}

__device__ __forceinline__ void put(float* p, float v, bool add) { *p = add ? *p + v : v; }

// this CTA's share of dW[j][k] = sum_r d[r][j] h[r][k] (N columns): a thread holds 8 x (N / 16) elements
template <int N>
__device__ __forceinline__ void bwd_weight(const float (&d)[kBwdRows][kMlpHidden], const float (&h)[kBwdRows][N],
                                           float* __restrict__ out, bool add) {
  constexpr int C = N / 16;                       // columns of a thread, in float4 groups 64 apart
  const int j0 = (threadIdx.x >> 4) * 8, k0 = (threadIdx.x & 15) * 4;
  float acc[8][C] = {};
#pragma unroll 2
  for (int r = 0; r < kBwdRows; ++r) {
    float dv[8], hv[C];
#pragma unroll
    for (int i = 0; i < 8; i += 4) *(float4*)&dv[i] = *(const float4*)&d[r][j0 + i];
#pragma unroll
    for (int c = 0; c < C; c += 4) *(float4*)&hv[c] = *(const float4*)&h[r][k0 + c * 16];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < C; ++c) acc[i][c] = fmaf(dv[i], hv[c], acc[i][c]);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int c = 0; c < C; ++c) put(out + (j0 + i) * N + k0 + (c / 4) * 64 + (c & 3), acc[i][c], add);
}

__global__ void __launch_bounds__(kBwdThreads, 1) k_bwd(int n, const __nv_bfloat16* __restrict__ pw,
    const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ act,
    const float* __restrict__ s, float* __restrict__ l, float* __restrict__ part, int np, MlpLayout L) {
  extern __shared__ __align__(16) unsigned char bsm_raw[];
  BwdSmem& S = *reinterpret_cast<BwdSmem*>(bsm_raw);
  constexpr int H = kMlpHidden;
  const int tid = threadIdx.x;
  for (int e = tid; e < H * H / 8; e += kBwdThreads) {
    ((uint4*)S.w3)[e] = __ldg((const uint4*)(pw + L.w3) + e);
    ((uint4*)S.w2)[e] = __ldg((const uint4*)(pw + L.w2) + e);
  }
  float* out = part + (size_t)blockIdx.x * np;
  for (int r0 = blockIdx.x * kBwdRows; r0 < n; r0 += gridDim.x * kBwdRows) {
    // every element of `out` belongs to one thread: a CTA's later tiles add to its first
    const bool add = r0 != (int)blockIdx.x * kBwdRows;
    const int nr = min(kBwdRows, n - r0);
    const float* h1 = act + (size_t)r0 * H;
    const float* h2 = h1 + (size_t)n * H;
    const float* h3 = h2 + (size_t)n * H;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);      // rows past n
    for (int e = tid; e < kBwdRows * H / 4; e += kBwdThreads) {
      const bool on = e / (H / 4) < nr;
      ((float4*)S.h1)[e] = on ? __ldg((const float4*)h1 + e) : z4;
      ((float4*)S.h2)[e] = on ? __ldg((const float4*)h2 + e) : z4;
      ((float4*)S.h3)[e] = on ? __ldg((const float4*)h3 + e) : z4;
    }
    for (int e = tid; e < kBwdRows * kMlpIn / 4; e += kBwdThreads)
      ((float4*)S.x)[e] = e / (kMlpIn / 4) < nr ? __ldg((const float4*)(x + (size_t)r0 * kMlpIn) + e) : z4;
    if (tid < kBwdRows) {   // dL/ds = (sigmoid(s) - y) / n and the per-sample loss softplus(s) - y s
      float g = 0.f;
      if (tid < nr) {
        const float z = s[r0 + tid], t = y[r0 + tid];
        const float sp = z > 0.f ? z + log1pf(expf(-z)) : log1pf(expf(z));
        const float sig = 1.f / (1.f + expf(-z));
        g = (sig - t) / (float)n;
        l[r0 + tid] = sp - t * z;
      }
      S.gs[tid] = g;
    }
    __syncthreads();
    for (int e = tid; e < kBwdRows * H; e += kBwdThreads) {
      const int r = e / H, j = e - r * H;
      S.d3[r][j] = S.h3[r][j] > 0.f ? S.gs[r] * __bfloat162float(pw[L.w4 + j]) : 0.f;
    }
    if (tid < H) {
      float acc = 0.f;
      for (int r = 0; r < kBwdRows; ++r) acc = fmaf(S.gs[r], S.h3[r][tid], acc);
      put(out + L.w4 + tid, acc, add);
    } else if (tid == H) {
      float acc = 0.f;
      for (int r = 0; r < kBwdRows; ++r) acc += S.gs[r];
      put(out + L.b4, acc, add);
    }
    __syncthreads();
    bwd_layer(S.d3, S.w3, S.h2, S.d2);
    __syncthreads();
    bwd_layer(S.d2, S.w2, S.h1, S.d1);
    __syncthreads();
    bwd_weight<H>(S.d3, S.h2, out + L.w3, add);
    bwd_weight<H>(S.d2, S.h1, out + L.w2, add);
    bwd_weight<kMlpIn>(S.d1, S.x, out + L.w1, add);
    for (int e = tid; e < 3 * H; e += kBwdThreads) {   // bias gradients: column sums of d1, d2, d3
      const int q = e / H, j = e - q * H;
      const float(*d)[H] = q == 0 ? S.d1 : q == 1 ? S.d2 : S.d3;
      float acc = 0.f;
      for (int r = 0; r < kBwdRows; ++r) acc += d[r][j];
      put(out + (q == 0 ? L.b1 : q == 1 ? L.b2 : L.b3) + j, acc, add);
    }
    __syncthreads();                                    // the next tile's rows overwrite these
  }
}

// g[p] = sum over the rows of `part` in row order, eight loads in flight; the last block sums the loss
constexpr int kSumGradThreads = 256;

__global__ void __launch_bounds__(kSumGradThreads) k_bwd_sum(int np, int nt, const float* __restrict__ part, int n,
    const float* __restrict__ l, float* __restrict__ g, double* __restrict__ loss) {
  if (blockIdx.x == gridDim.x - 1) {
    __shared__ double red[32];
    double acc = 0.0;
    for (int i = threadIdx.x; i < n; i += kSumGradThreads) acc += (double)l[i];
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
      double v = threadIdx.x < (kSumGradThreads >> 5) ? red[threadIdx.x] : 0.0;
      v = warp_sum(v);
      if (threadIdx.x == 0) *loss = v / (double)n;
    }
    return;
  }
  const int p = blockIdx.x * kSumGradThreads + threadIdx.x;
  if (p >= np) return;
  float acc = 0.f;
  int t = 0;
  for (; t + 8 <= nt; t += 8) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = part[(size_t)(t + u) * np + p];
#pragma unroll
    for (int u = 0; u < 8; ++u) acc += v[u];
  }
  for (; t < nt; ++t) acc += part[(size_t)t * np + p];
  g[p] = acc;
}

__global__ void k_to_bf16(int n, const float* __restrict__ src, __nv_bfloat16* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = __float2bfloat16_rn(src[i]);
}

__global__ void k_adam(int n, float lr, float b1, float b2, float eps, float c1, float c2, float* __restrict__ w,
                       float* __restrict__ m, float* __restrict__ v, const float* __restrict__ g,
                       __nv_bfloat16* __restrict__ wb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float upd = lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[i] -= upd;
  wb[i] = __float2bfloat16_rn(w[i]);
}

// ---- the forward pass on the tensor cores (tcgen05, kind::tf32) -----------
// One CTA per 128 samples, 128 threads.  The three hidden layers are 128 x 128 x K
// MMAs (K = 64, 128, 128) with the samples on the M side: A = the layer's input
// rows, B = the weight matrix [out][in], both K-major in 128-byte-swizzled shared
// memory (32 TF32 per 128-byte row, one 16 KB atom per 32 of K).  The BF16 weights
// are exact in TF32; the inputs are rounded to TF32 (nearest, ties away) as they
// are staged.  The FP32 accumulator (TMEM, 128 lanes x 128 columns) gets the FP32
// bias and the ReLU in the epilogue, which stores the activation in FP32 (the
// backward pass reads it) and stages it, rounded, as the next layer's A.  The
// output layer is a 128-term FP32 dot product per sample, in column order.  Every
// mbarrier wait has an iteration limit; on expiry the kernel sets *err and skips.
constexpr int kFwdRows = 128;
constexpr int kFwdAtoms = kMlpHidden / 32;            // K atoms of a 128-wide input

struct FwdSmem {
  uint32_t a[kFwdAtoms][kFwdRows * 32];               // layer input, TF32 bits, 4 x 16 KB
  uint32_t b[kFwdAtoms][kMlpHidden * 32];             // weights, TF32 bits, 4 x 16 KB
  uint64_t bar;
  uint32_t tmem_base;
};
constexpr size_t kFwdSmemBytes = sizeof(FwdSmem) + 1024;

// instruction descriptor: kind::tf32, D = F32, A = B = TF32, both K-major, M = 128, N = 128
__host__ __device__ constexpr uint32_t idesc_tf32() {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(kMlpHidden >> 3) << 17) | ((uint32_t)(kFwdRows >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
  const uint32_t idesc = idesc_tf32();
  const uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      :
      : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(z), "r"(z), "r"(z), "r"(z));
}

__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}

// element (row, k) of a K-major swizzled operand of `atoms` x 16 KB: 32 TF32 per atom row
__device__ __forceinline__ uint32_t* tf32_slot(uint32_t (*op)[kFwdRows * 32], int row, int k) {
  const int atom = k >> 5, kk = k & 31;
  return (uint32_t*)((unsigned char*)op[atom] + tc::swz(row, kk >> 2)) + (kk & 3);
}

// Operand staging with 16-byte loads, kStageBatch in flight per thread: x rows (FP32, 4 per
// load) and weight rows (BF16, 8 per load) into the swizzled TF32 layout; every group of four
// consecutive k lands in one 16-byte chunk of a row.  Unaligned sources take the scalar loop.
constexpr int kStageBatch = 16;

__device__ __forceinline__ void stage_x(uint32_t (*a)[kFwdRows * 32], const float* __restrict__ x, int r0, int n,
                                        int tid) {
  constexpr int Q = kMlpIn / 4, TOT = kFwdRows * Q;            // float4 per row, per tile
  if (((uintptr_t)x & 15) == 0) {
#pragma unroll 1
    for (int e0 = 0; e0 < TOT; e0 += kStageBatch * kFwdRows) {
      float4 v[kStageBatch];
#pragma unroll
      for (int u = 0; u < kStageBatch; ++u) {
        const int e = e0 + u * kFwdRows + tid, row = e / Q;
        v[u] = (e < TOT && r0 + row < n) ? __ldg((const float4*)(x + (size_t)(r0 + row) * kMlpIn) + (e - row * Q))
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < kStageBatch; ++u) {
        const int e = e0 + u * kFwdRows + tid, row = e / Q;
        if (e < TOT)
          *(uint4*)tf32_slot(a, row, (e - row * Q) * 4) =
              make_uint4(to_tf32(v[u].x), to_tf32(v[u].y), to_tf32(v[u].z), to_tf32(v[u].w));
      }
    }
  } else {
    for (int e = tid; e < kFwdRows * kMlpIn; e += kFwdRows) {
      const int row = e / kMlpIn, k = e - row * kMlpIn;
      const float v = (r0 + row < n) ? x[(size_t)(r0 + row) * kMlpIn + k] : 0.f;
      *tf32_slot(a, row, k) = to_tf32(v);
    }
  }
}

template <int K>
__device__ __forceinline__ void stage_w(uint32_t (*b)[kMlpHidden * 32], const __nv_bfloat16* __restrict__ w, int tid) {
  constexpr int Q = K / 8, TOT = kMlpHidden * Q;               // 16-byte groups per row, per matrix
  if (((uintptr_t)w & 15) == 0) {
#pragma unroll 1
    for (int e0 = 0; e0 < TOT; e0 += kStageBatch * kFwdRows) {
      uint4 v[kStageBatch];
#pragma unroll
      for (int u = 0; u < kStageBatch; ++u) {
        const int e = e0 + u * kFwdRows + tid;
        v[u] = e < TOT ? __ldg((const uint4*)w + e) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < kStageBatch; ++u) {
        const int e = e0 + u * kFwdRows + tid, o = e / Q, k = (e - o * Q) * 8;
        if (e < TOT) {
          // a BF16 is the high half of its FP32 (and TF32) pattern
          const uint32_t p[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
          *(uint4*)tf32_slot(b, o, k) = make_uint4(p[0] << 16, p[0] & 0xffff0000u, p[1] << 16, p[1] & 0xffff0000u);
          *(uint4*)tf32_slot(b, o, k + 4) = make_uint4(p[2] << 16, p[2] & 0xffff0000u, p[3] << 16, p[3] & 0xffff0000u);
        }
      }
    }
  } else {
    for (int e = tid; e < kMlpHidden * K; e += kFwdRows) {
      const int o = e / K, k = e - o * K;
      *tf32_slot(b, o, k) = __float_as_uint(__bfloat162float(w[e]));
    }
  }
}

__global__ void __launch_bounds__(kFwdRows, 1) k_mlp_fwd_tc(const __nv_bfloat16* __restrict__ pw,
    const float* __restrict__ pf, const float* __restrict__ x, int n, float* __restrict__ act,
    float* __restrict__ logits, int* __restrict__ err, MlpLayout L) {
  using namespace tc;
  extern __shared__ __align__(1024) unsigned char fsm_raw[];
  FwdSmem& S = *reinterpret_cast<FwdSmem*>((void*)(((uintptr_t)fsm_raw + 1023) & ~(uintptr_t)1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r0 = blockIdx.x * kFwdRows;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)),
                 "r"(kMlpHidden));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    mbar_init(&S.bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // layer 1 input: x rows, rounded to TF32 (rows past n are zero)
  stage_x(S.a, x, r0, n, tid);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S.tmem_base;
  bool ok = true;
  const int row = r0 + warp * 32 + lane;              // this thread's sample (TMEM lane)
  float out = 0.f;
  const int woff[3] = {L.w1, L.w2, L.w3}, boff[3] = {L.b1, L.b2, L.b3}, kin[3] = {kMlpIn, kMlpHidden, kMlpHidden};
  for (int layer = 0; layer < 3; ++layer) {
    const int K = kin[layer];
    // weights [out][K] (BF16, exact in TF32) as the B operand
    if (K == kMlpIn) stage_w<kMlpIn>(S.b, pw + woff[layer], tid);
    else stage_w<kMlpHidden>(S.b, pw + woff[layer], tid);
    fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      for (int atom = 0; atom < K / 32; ++atom) {
        const uint64_t da = smem_desc(smem_u32(S.a[atom])), db = smem_desc(smem_u32(S.b[atom]));
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)   // K = 8 TF32 (32 bytes) per MMA
          mma_tf32(tmem, da + (uint64_t)(ks * 2), db + (uint64_t)(ks * 2), (atom > 0 || ks > 0) ? 1u : 0u);
      }
      mma_commit(&S.bar);
    }
    const bool done = mbar_wait(&S.bar, (uint32_t)(layer & 1));
    ok = __syncthreads_and(done && ok) != 0;
    if (!ok) break;
    tc_fence_after();
    float* h = act ? act + (size_t)layer * n * kMlpHidden : nullptr;
    for (int c0 = 0; c0 < kMlpHidden; c0 += 32) {
      uint32_t v[32];
      tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        const int col = c0 + e;
        const float z = fmaxf(__uint_as_float(v[e]) + pf[boff[layer] + col], 0.f);
        if (act && row < n) h[(size_t)row * kMlpHidden + col] = z;
        if (layer < 2) *tf32_slot(S.a, warp * 32 + lane, col) = to_tf32(z);
        else out = fmaf(z, __bfloat162float(pw[L.w4 + col]), out);
      }
    }
    tc_fence_before();
    __syncthreads();
  }
  if (ok && row < n) logits[row] = out + pf[L.b4];
  if (!ok) {
    if (tid == 0 && err) atomicOr(err, kErrTimeout);
    mbar_wait(&S.bar, 0u);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kMlpHidden));
}

}  // namespace

// ---- shared by the engine: inference over the voxels of a frame ----------

MlpLayout mlp_layout() {
  MlpLayout L;
  L.w1 = 0;
  L.b1 = L.w1 + kMlpHidden * kMlpIn;
  L.w2 = L.b1 + kMlpHidden;
  L.b2 = L.w2 + kMlpHidden * kMlpHidden;
  L.w3 = L.b2 + kMlpHidden;
  L.b3 = L.w3 + kMlpHidden * kMlpHidden;
  L.w4 = L.b3 + kMlpHidden;
  L.b4 = L.w4 + kMlpHidden;
  L.n = L.b4 + 1;
  return L;
}

// Biases stay FP32 (the FP32 copy of the parameters is passed as `pf`); the
// weight matrices are read as BF16.  act: [3][n][128] hidden activations for the
// backward pass, or NULL (inference); logits: [n].  err (device, may be NULL):
// kErrTimeout is or-ed in if a tensor-core wait gave up.
void mlp_forward(const __nv_bfloat16* pw, const float* pf, const float* x, int n, float* act, float* logits,
                 int* err, cudaStream_t s) {
  if (n <= 0) return;
  raise_smem_limit(k_mlp_fwd_tc, kFwdSmemBytes);
  k_mlp_fwd_tc<<<(n + kFwdRows - 1) / kFwdRows, kFwdRows, kFwdSmemBytes, s>>>(pw, pf, x, n, act, logits, err,
                                                                             mlp_layout());
}

int mlp_forward_launches() { return 1; }

}  // namespace erm

// ---- the trainer (C-ABI) -----------------------------------------------------

using namespace erm;

struct ermod_mlp {
  int device = 0, max_batch = 0;
  cudaStream_t st = nullptr;
  float *w = nullptr, *m = nullptr, *v = nullptr, *g = nullptr;   // FP32 master, Adam moments, gradient
  __nv_bfloat16* wb = nullptr;                                     // BF16 weights used by every pass
  float *x = nullptr, *y = nullptr, *act = nullptr, *s = nullptr, *l = nullptr;
  float* part = nullptr;         // [CTAs of a full batch][np] shares of the gradient
  double* loss = nullptr;        // behind the gradient in g's allocation, so one copy brings back both
  int* dev_err = nullptr;        // behind the loss: set by the tensor-core forward if a wait gave up
  unsigned char* h_out = nullptr;   // pinned image of g's allocation
  long long t = 0;
  std::string err;
};

namespace {
// g's allocation: np gradient floats, the loss (FP64), the tensor-core forward's error word
size_t loss_off() { return sizeof(float) * (((size_t)mlp_layout().n + 1) & ~(size_t)1); }
size_t out_bytes() { return loss_off() + sizeof(double) + sizeof(int); }

// Bring `bytes` from `off` of that allocation to its pinned image, wait for the stream and take the
// error word (cleared for the next call where set).
int fetch_out(ermod_mlp* p, size_t off, size_t bytes) {
  if (cudaMemcpyAsync(p->h_out + off, (unsigned char*)p->g + off, bytes, cudaMemcpyDeviceToHost, p->st) != cudaSuccess ||
      cudaStreamSynchronize(p->st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
    return ERMOD_ERR_CUDA;
  int e = 0;
  std::memcpy(&e, p->h_out + loss_off() + sizeof(double), sizeof(int));
  if (e == 0) return ERMOD_OK;
  cudaMemset(p->dev_err, 0, sizeof(int));
  p->err = "tc_wait";
  return ERMOD_ERR_CUDA;
}

void mlp_free(ermod_mlp* p) {
  void* ptrs[] = {p->w, p->m, p->v, p->g, p->wb, p->x, p->y, p->act, p->s, p->l, p->part};
  for (void* q : ptrs)
    if (q) cudaFree(q);
  if (p->h_out) cudaFreeHost(p->h_out);
  if (p->st) cudaStreamDestroy(p->st);
}

// x and y (host) into the device batch buffers
int stage(ermod_mlp* p, const float* x, const float* y, int n) {
  if (cudaMemcpyAsync(p->x, x, sizeof(float) * (size_t)n * kMlpIn, cudaMemcpyHostToDevice, p->st) != cudaSuccess)
    return ERMOD_ERR_CUDA;
  if (y && cudaMemcpyAsync(p->y, y, sizeof(float) * n, cudaMemcpyHostToDevice, p->st) != cudaSuccess)
    return ERMOD_ERR_CUDA;
  return ERMOD_OK;
}

// forward + loss + backward into p->g for a staged batch of n samples
int backward(ermod_mlp* p, int n) {
  const MlpLayout L = mlp_layout();
  cudaStream_t s = p->st;
  if (raise_smem_limit(k_bwd, sizeof(BwdSmem)) != cudaSuccess) return ERMOD_ERR_CUDA;
  mlp_forward(p->wb, p->w, p->x, n, p->act, p->s, p->dev_err, s);
  const int nt = bwd_parts(n);
  k_bwd<<<nt, kBwdThreads, sizeof(BwdSmem), s>>>(n, p->wb, p->x, p->y, p->act, p->s, p->l, p->part, L.n, L);
  k_bwd_sum<<<(L.n + kSumGradThreads - 1) / kSumGradThreads + 1, kSumGradThreads, 0, s>>>(L.n, nt, p->part, n, p->l,
                                                                                        p->g, p->loss);
  return ERMOD_OK;
}
}  // namespace

extern "C" {

int32_t ermod_mlp_create(ermod_mlp** out, int32_t device, int32_t max_batch, const float* init_params) {
  if (!out || max_batch <= 0 || !init_params) return ERMOD_ERR_ARG;
  *out = nullptr;
  ermod_mlp* p = new ermod_mlp();
  p->device = device;
  p->max_batch = max_batch;
  const int np = mlp_layout().n;
  const size_t B = (size_t)max_batch;
  auto A = [&](auto** q, size_t n) { return cudaMalloc((void**)q, sizeof(**q) * std::max<size_t>(n, 1)); };
  bool ok = cudaSetDevice(device) == cudaSuccess && cudaStreamCreateWithFlags(&p->st, cudaStreamNonBlocking) == 0 &&
            A(&p->w, np) == 0 && A(&p->m, np) == 0 && A(&p->v, np) == 0 &&
            cudaMalloc((void**)&p->g, out_bytes()) == cudaSuccess &&
            cudaMallocHost((void**)&p->h_out, out_bytes()) == cudaSuccess &&
            A(&p->wb, np) == 0 && A(&p->x, B * kMlpIn) == 0 && A(&p->y, B) == 0 &&
            A(&p->act, 3 * B * kMlpHidden) == 0 && A(&p->s, B) == 0 && A(&p->l, B) == 0 &&
            A(&p->part, (size_t)bwd_parts(max_batch) * np) == 0;
  if (ok) {
    p->loss = (double*)((unsigned char*)p->g + loss_off());
    p->dev_err = (int*)(p->loss + 1);
    ok = cudaMemcpyAsync(p->w, init_params, sizeof(float) * np, cudaMemcpyHostToDevice, p->st) == cudaSuccess &&
         cudaMemsetAsync(p->m, 0, sizeof(float) * np, p->st) == cudaSuccess &&
         cudaMemsetAsync(p->v, 0, sizeof(float) * np, p->st) == cudaSuccess &&
         cudaMemsetAsync(p->dev_err, 0, sizeof(int), p->st) == cudaSuccess;
    k_to_bf16<<<(np + 255) / 256, 256, 0, p->st>>>(np, p->w, p->wb);
    ok = ok && cudaStreamSynchronize(p->st) == cudaSuccess && cudaGetLastError() == cudaSuccess;
  }
  if (!ok) {
    mlp_free(p);
    delete p;
    return ERMOD_ERR_CUDA;
  }
  *out = p;
  return ERMOD_OK;
}

int32_t ermod_mlp_nparams(void) { return mlp_layout().n; }

// logits of n samples x[n][64] (host) with the current BF16 weights
int32_t ermod_mlp_forward(ermod_mlp* p, const float* x, int32_t n, float* logits) {
  if (!p || !x || !logits || n <= 0 || n > p->max_batch) return ERMOD_ERR_ARG;
  if (cudaSetDevice(p->device) != cudaSuccess) return ERMOD_ERR_CUDA;
  int rc = stage(p, x, nullptr, n);
  if (rc != ERMOD_OK) return rc;
  mlp_forward(p->wb, p->w, p->x, n, p->act, p->s, p->dev_err, p->st);
  if (cudaMemcpyAsync(logits, p->s, sizeof(float) * n, cudaMemcpyDeviceToHost, p->st) != cudaSuccess)
    return ERMOD_ERR_CUDA;
  return fetch_out(p, loss_off(), out_bytes() - loss_off());
}

// the hidden activations [3][n][128] (FP32, after bias and ReLU) of the last
// forward or gradient pass over n samples
int32_t ermod_mlp_activations(ermod_mlp* p, int32_t n, float* act) {
  if (!p || !act || n <= 0 || n > p->max_batch) return ERMOD_ERR_ARG;
  if (cudaSetDevice(p->device) != cudaSuccess) return ERMOD_ERR_CUDA;
  if (cudaMemcpyAsync(act, p->act, sizeof(float) * 3 * (size_t)n * kMlpHidden, cudaMemcpyDeviceToHost, p->st) !=
          cudaSuccess ||
      cudaStreamSynchronize(p->st) != cudaSuccess)
    return ERMOD_ERR_CUDA;
  return ERMOD_OK;
}

// mean loss and its gradient (FP32, ERMOD_MLP_NPARAMS) for a batch, no update
int32_t ermod_mlp_gradients(ermod_mlp* p, const float* x, const float* y, int32_t n, float* grad, double* loss) {
  if (!p || !x || !y || n <= 0 || n > p->max_batch) return ERMOD_ERR_ARG;
  if (cudaSetDevice(p->device) != cudaSuccess) return ERMOD_ERR_CUDA;
  int rc = stage(p, x, y, n);
  if (rc != ERMOD_OK) return rc;
  if ((rc = backward(p, n)) != ERMOD_OK) return rc;
  const size_t off = grad ? 0 : loss_off();
  if ((rc = fetch_out(p, off, out_bytes() - off)) != ERMOD_OK) return rc;
  if (grad) std::memcpy(grad, p->h_out, sizeof(float) * mlp_layout().n);
  if (loss) std::memcpy(loss, p->h_out + loss_off(), sizeof(double));
  return ERMOD_OK;
}

// one Adam step on a batch; returns the batch's mean loss before the step
int32_t ermod_mlp_train_step(ermod_mlp* p, const float* x, const float* y, int32_t n, float lr, double* loss) {
  if (!p || !x || !y || n <= 0 || n > p->max_batch || !(lr > 0.f)) return ERMOD_ERR_ARG;
  if (cudaSetDevice(p->device) != cudaSuccess) return ERMOD_ERR_CUDA;
  int rc = stage(p, x, y, n);
  if (rc != ERMOD_OK) return rc;
  if ((rc = backward(p, n)) != ERMOD_OK) return rc;
  ++p->t;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - (float)std::pow((double)b1, (double)p->t), c2 = 1.f - (float)std::pow((double)b2, (double)p->t);
  const int np = mlp_layout().n;
  k_adam<<<(np + 255) / 256, 256, 0, p->st>>>(np, lr, b1, b2, 1e-8f, c1, c2, p->w, p->m, p->v, p->g, p->wb);
  if ((rc = fetch_out(p, loss_off(), out_bytes() - loss_off())) != ERMOD_OK) return rc;
  if (loss) std::memcpy(loss, p->h_out + loss_off(), sizeof(double));
  return ERMOD_OK;
}

// FP32 master parameters (host)
int32_t ermod_mlp_get_params(ermod_mlp* p, float* params) {
  if (!p || !params) return ERMOD_ERR_ARG;
  if (cudaSetDevice(p->device) != cudaSuccess) return ERMOD_ERR_CUDA;
  if (cudaMemcpyAsync(params, p->w, sizeof(float) * mlp_layout().n, cudaMemcpyDeviceToHost, p->st) != cudaSuccess ||
      cudaStreamSynchronize(p->st) != cudaSuccess)
    return ERMOD_ERR_CUDA;
  return ERMOD_OK;
}

void ermod_mlp_destroy(ermod_mlp* p) {
  if (!p) return;
  cudaSetDevice(p->device);
  if (p->st) cudaStreamSynchronize(p->st);
  mlp_free(p);
  delete p;
}

}  // extern "C"

namespace erm {
void launch_to_bf16(int n, const float* src, __nv_bfloat16* dst, cudaStream_t s) {
  k_to_bf16<<<(n + 255) / 256, 256, 0, s>>>(n, src, dst);
}
}  // namespace erm
