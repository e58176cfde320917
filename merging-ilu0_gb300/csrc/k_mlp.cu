// Learned ParILU(0) warm start: a per-nonzero MLP (9 -> 64 -> 64 -> 1, GELU in
// its tanh form, BF16 weights, FP32 accumulation) that predicts the converged
// ParILU factors, trained on the GPU by these kernels.  No counterpart in the
// reference.  The 64-wide GEMMs run on the Blackwell tensor cores (tcgen05.mma
// with BF16 operands in shared memory and FP32 accumulators in tensor memory,
// k_tc.cuh; activations and gradients split into BF16 high + low parts so the
// products keep FP32-level precision): in training (k_mlp_train) the forward
// 64x64 layer, the backward dh1 = dpre2 W2 and the weight gradient
// dW2 = dpre2^T H1, with the accurate tanh on the CUDA cores; in inference
// (k_mlp_warm) the 64x64 layer, with the hardware tanh approximation.
//
// Features of nonzero (i, j) of system s, all scaled by d = |a_ii|:
//   a_ij, a_ii, a_jj, ||A(i,:)||_2, ||A(:,j)||_2 (column over the structurally
//   symmetric part), level(i) / (levels-1), sign(j - i), and the first-order
//   Schur corrections c_i, c_j with c_r = sum_{k<r} a_rk a_kr / a_kk.
// Output y is a relative correction of a first-order estimate of the factor
// ratio lu_ij / a_ij:  below the diagonal 1 / (a_jj - c_j), on it
// (a_ii - c_i) / a_ii, above it 1;  warm start lu0_ij = a_ij * base * (1 + y).
// Training target: y* = lu*_ij / (a_ij * base) - 1 with lu* the converged
// ParILU(0) factors the solver generates; loss = mean (y - y*)^2.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "bilu_internal.h"
#include "k_intfp.cuh"
#include "k_tc.cuh"

namespace bilu {
namespace {

constexpr int NF = kMlpFeatures;
constexpr int H = kMlpHidden;
constexpr int OW1 = 0, OB1 = H * NF, OW2 = OB1 + H, OB2 = OW2 + H * H, OW3 = OB2 + H, OB3 = OW3 + H;
static_assert(OB3 + 1 == kMlpParams, "parameter layout");

constexpr unsigned kFull = 0xffffffffu;
// polls of an mbarrier before a tensor-core round counts as failed (it completes in microseconds)
constexpr uint32_t kWaitLimit = 1u << 24;

// GELU, tanh form: 0.5 x (1 + tanh(k (x + c x^3))), k = sqrt(2/pi), c = 0.044715
constexpr float kGk = 0.7978845608028654f, kGc = 0.044715f;
__device__ __forceinline__ float gelu(float x) {
  const float t = tanhf(kGk * fmaf(kGc * x, x * x, x));
  return 0.5f * x * (1.0f + t);
}
__device__ __forceinline__ float gelu_d(float x) {
  const float t = tanhf(kGk * fmaf(kGc * x, x * x, x));
  return 0.5f * (1.0f + t) + 0.5f * x * (1.0f - t * t) * kGk * fmaf(3.0f * kGc, x * x, 1.0f);
}
__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float gelu_fast(float x) {
  return 0.5f * x * (1.0f + tanh_approx(kGk * fmaf(kGc * x, x * x, x)));
}

// per (system, row): row 2-norm, column 2-norm, first-order Schur correction
__global__ void k_rowstats(const DevPattern P, int nsys, const double* __restrict__ A, float* __restrict__ rown,
                           float* __restrict__ coln, float* __restrict__ corr) {
  const int s = blockIdx.x;
  if (s >= nsys) return;
  // FP32 throughout (the features are FP32): FP64 division and square root
  // are long instruction sequences on this part's FP64 pipe, where hardware
  // conversions run too (88 % of it at 4096 7x7x7 systems, 53 us)
  const double* As = A + (size_t)s * P.nnz;
  for (int i = threadIdx.x; i < P.n; i += blockDim.x) {
    const int b = P.rp[i], e = P.rp[i + 1], d = P.diag[i];
    float rn = 0.0f, cn = 0.0f, c = 0.0f;
    for (int k = b; k < e; ++k) {
      const float a = ifp::f32(As[k]);
      rn = fmaf(a, a, rn);
      const int t = P.tpos[k];
      if (t >= 0) {
        const float at = ifp::f32(As[t]);
        cn = fmaf(at, at, cn);
        if (k < d) c = fmaf(a, at / ifp::f32(As[P.diag[P.ci[k]]]), c);
      }
    }
    rown[(size_t)s * P.n + i] = sqrtf(rn);
    coln[(size_t)s * P.n + i] = sqrtf(cn);
    corr[(size_t)s * P.n + i] = c;
  }
}

struct Feat {
  float f[NF];
  float base;
  double a;
};

// Features in FP32 from one reciprocal (FP64 divisions are expensive on this
// part); base = first-order estimate of the factor ratio (FP32).
__device__ __forceinline__ Feat features(const DevPattern& P, int s, int e, const double* __restrict__ A,
                                         const float* __restrict__ rown, const float* __restrict__ coln,
                                         const float* __restrict__ corr) {
  Feat r;
  const int i = P.row_of[e], j = P.ci[e];
  const double* As = A + (size_t)s * P.nnz;
  const double aij = As[e];
  const float fij = ifp::f32(aij), fii = ifp::f32(As[P.diag[i]]), fjj = ifp::f32(As[P.diag[j]]);
  const float inv = 1.0f / (fii != 0.0f ? fabsf(fii) : 1.0f);
  const float ci_ = corr[(size_t)s * P.n + i], cj = corr[(size_t)s * P.n + j];
  r.f[0] = fij * inv;
  r.f[1] = fii * inv;
  r.f[2] = fjj * inv;
  r.f[3] = rown[(size_t)s * P.n + i] * inv;
  r.f[4] = coln[(size_t)s * P.n + j] * inv;
  r.f[5] = P.nlev_lo > 1 ? (float)P.row_lev[i] / (float)(P.nlev_lo - 1) : 0.0f;
  r.f[6] = j < i ? -1.0f : (j > i ? 1.0f : 0.0f);
  r.f[7] = ci_ * inv;
  r.f[8] = cj * inv;
  r.a = aij;
  float base = 1.0f;
  if (j < i) {
    const float den = fjj - cj;
    base = den != 0.0f ? 1.0f / den : (fjj != 0.0f ? 1.0f / fjj : 1.0f);
  } else if (j == i) {
    base = fii != 0.0f ? (fii - ci_) / fii : 1.0f;
  }
  r.base = base;
  return r;
}

// parameters (BF16) staged into shared memory as FP32
__device__ __forceinline__ void stage_params(const __nv_bfloat16* __restrict__ pbf, float* sp) {
  for (int k = threadIdx.x; k < kMlpParams; k += blockDim.x) sp[k] = __bfloat162float(pbf[k]);
}

// forward of one sample on CUDA cores; h1 / g1 / pre2 optionally stored (row of stride 65)
__device__ __forceinline__ float mlp_forward(const float* sp, const float* x, float* h1row, float* g1row,
                                             float* p2row) {
  float h[H];
#pragma unroll 4
  for (int u = 0; u < H; ++u) {
    float acc = sp[OB1 + u];
#pragma unroll
    for (int k = 0; k < NF; ++k) acc = fmaf(sp[OW1 + u * NF + k], x[k], acc);
    h[u] = gelu(acc);
    if (h1row) {
      h1row[u] = h[u];
      g1row[u] = gelu_d(acc);
    }
  }
  float out = sp[OB3];
  for (int u = 0; u < H; ++u) {
    float acc = sp[OB2 + u];
    const float4* w = reinterpret_cast<const float4*>(sp + OW2 + u * H);
#pragma unroll
    for (int v4 = 0; v4 < H / 4; ++v4) {
      const float4 q = w[v4];
      acc = fmaf(q.x, h[4 * v4 + 0], acc);
      acc = fmaf(q.y, h[4 * v4 + 1], acc);
      acc = fmaf(q.z, h[4 * v4 + 2], acc);
      acc = fmaf(q.w, h[4 * v4 + 3], acc);
    }
    if (p2row) p2row[u] = acc;
    out = fmaf(sp[OW3 + u], gelu(acc), out);
  }
  return out;
}

uint64_t __host__ __device__ __forceinline__ mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

constexpr int TB = 128;  // samples (threads) per training block
constexpr int LD = H + 1;

// BF16 high part of x and the BF16 of what is left (x = hi + lo to about 16 bits)
__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16& hi, __nv_bfloat16& lo) {
  hi = __float2bfloat16_rn(x);
  lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}

// Sum over the 32 lanes of a warp of 32 values per lane, scattered: lane l
// returns the warp's sum of v[l] (recursive halving, 31 shuffles).
__device__ __forceinline__ float warp_reduce_scatter32(const float (&v)[32]) {
  const int lane = threadIdx.x & 31;
  float a[16];
  {
    const bool up = lane & 16;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float mine = up ? v[i + 16] : v[i], send = up ? v[i] : v[i + 16];
      a[i] = mine + __shfl_xor_sync(kFull, send, 16);
    }
  }
#pragma unroll
  for (int w = 8; w >= 1; w >>= 1) {
    const bool up = lane & w;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float mine = up ? a[i + w] : a[i], send = up ? a[i] : a[i + w];
      a[i] = mine + __shfl_xor_sync(kFull, send, w);
    }
  }
  return a[0];
}

// Training block layout (dynamic shared memory, 1024-byte aligned):
//   A1   [128][64] BF16 hi, lo    K-major: H1 (layer-1 activations), later dpre2
//   BT   [64][128] BF16 hi, lo    K-major: H1^T (B operand of dW2, K = samples)
//   AT   [128][128] BF16          K-major: dpre2^T, rows 0..63 high parts, 64..127 low parts
//   BW   [64][64] BF16            K-major: W2 (row u = output unit)
//   BWT  [64][64] BF16            K-major: W2^T (row v = input unit)
//   W1   [64][12] FP32            W1[v][0..8], b1[v], 0, 0
//   BWV  [64] float2              (b2[u], w3[u])
//   X    [128][9] FP32            features
//   G1   [128][65] FP32           gelu'(pre1), later dpre1
//   RED  [3][4][64] FP32          per-warp sums of db2, dW3, db1
constexpr int TR_A1 = 0, TR_BT = TR_A1 + 2 * TB * H * 2, TR_AT = TR_BT + 2 * H * TB * 2, TR_BW = TR_AT + TB * TB * 2;
constexpr int TR_BWT = TR_BW + H * H * 2, TR_W1 = TR_BWT + H * H * 2, TR_BWV = TR_W1 + H * 12 * 4;
constexpr int TR_X = TR_BWV + H * 8, TR_G1 = TR_X + TB * NF * 4, TR_RED = TR_G1 + TB * LD * 4;
constexpr int TR_SMEM = TR_RED + 3 * 4 * H * 4;
constexpr uint32_t kTrainTmemCols = 256;  // D1 pre2 | D2 dh1 | D3, D4 the two halves of dW2
static_assert(TR_W1 % 16 == 0 && TR_X % 16 == 0, "aligned blocks");
constexpr int kTrainRow = (kMlpParams + 1 + 3) & ~3;  // floats of a block's row: the gradient, the loss
static_assert(OW2 % 4 == 0 && H * LD * 4 <= TB * TB * 2, "dW2 rows");

// One forward + backward pass over a block of 128 samples (thread = sample) with
// the three 64-wide GEMMs on the tensor cores (tcgen05.mma, BF16 operands
// split into high and low parts, FP32 accumulators in TMEM):
//   forward   pre2 = H1 W2^T                 (M = 128 samples, N = 64, K = 64)
//   backward  dh1  = dpre2 W2                (M = 128 samples, N = 64, K = 64)
//             dW2  = dpre2^T H1              (M = 128: the 64 units' high and low
//                                             parts stacked, N = 64, K = 128 samples)
// Layer 1, the activations and the output layer run on the CUDA cores in FP32
// with the accurate tanh.  Per-unit sums over the block (db1, db2, dW3) are
// reduce-scattered across each warp; dW1 is reduced over the block in shared
// memory; the block's share of the gradient and of the loss is added to row
// blockIdx.x / 2 of `rows` (kTrainRow floats, zero before: the gradient, then
// the loss), which k_grad_sum adds up in a fixed order.  Two shares per
// row, because the sum of zero and two numbers is the same in either order, and
// half the rows keep a small model's memory within one of the driver's 2 MB
// chunks (a new one costs 0.17 ms per model: create, 8 steps of 9000 samples
// and destroy 0.59 ms with a row per block, 0.40 with this).  (Additions of
// every block to one gradient gave other bits on every run: a parameter on a
// BF16 rounding boundary then moves the losses of the steps that follow, by
// 1e-7 to 5e-4 over 40 steps.)  Samples: explicit global entry indices
// (s*nnz+e) or, when idx == NULL, hashed from (seed, sample number).  A
// tensor-core round that does not complete within the bounded wait adds NaN to
// the loss and ends the block.
__global__ void __launch_bounds__(TB) k_mlp_train(const DevPattern P, int nsys, const double* __restrict__ A,
                                                  const double* __restrict__ LUt, const float* __restrict__ rown,
                                                  const float* __restrict__ coln, const float* __restrict__ corr,
                                                  const __nv_bfloat16* __restrict__ pbf, int nsample,
                                                  const int* __restrict__ idx, uint64_t seed, float scale,
                                                  long long first, float* __restrict__ rows) {
  extern __shared__ __align__(1024) unsigned char smt[];
  __shared__ uint64_t s_mbar;
  __shared__ uint32_t s_tmem;
  __shared__ float s_loss[TB / 32], s_do[TB / 32];
  __shared__ int s_fail;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  float* X = reinterpret_cast<float*>(smt + TR_X);
  float* G1 = reinterpret_cast<float*>(smt + TR_G1);
  float* RED = reinterpret_cast<float*>(smt + TR_RED);
  // ---- weights
  {
    const uint4* w2g = reinterpret_cast<const uint4*>(pbf + OW2);
    for (int k = t; k < H * 8; k += TB) {
      const int u = k >> 3, c = k & 7;
      *reinterpret_cast<uint4*>(smt + TR_BW + tc::kmajor_off(u, 8 * c, H)) = w2g[k];
    }
    for (int k = t; k < H * H; k += TB) {  // W2^T: element (v, u) = W2[u][v]
      const int u = k >> 6, v = k & 63;
      *reinterpret_cast<__nv_bfloat16*>(smt + TR_BWT + tc::kmajor_off(v, u, H)) = pbf[OW2 + k];
    }
    float* w1 = reinterpret_cast<float*>(smt + TR_W1);
    for (int k = t; k < H * 12; k += TB) {
      const int v = k / 12, c = k % 12;
      w1[k] = c < NF ? __bfloat162float(pbf[OW1 + v * NF + c]) : (c == NF ? __bfloat162float(pbf[OB1 + v]) : 0.0f);
    }
    float2* bwv = reinterpret_cast<float2*>(smt + TR_BWV);
    for (int u = t; u < H; u += TB) bwv[u] = make_float2(__bfloat162float(pbf[OB2 + u]), __bfloat162float(pbf[OW3 + u]));
  }
  if (t == 0) {
    tc::mbar_init(&s_mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_fail = 0;
  }
  if (warp == 0) tc::alloc(&s_tmem, kTrainTmemCols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = s_tmem;
  const uint32_t trow = tmem + ((uint32_t)(32 * warp) << 16);
  const float4* w1v = reinterpret_cast<const float4*>(smt + TR_W1);
  const float2* bwv = reinterpret_cast<const float2*>(smt + TR_BWV);
  const float b3 = __bfloat162float(pbf[OB3]);
  // ---- sample, features, target
  const long long q = first + (long long)blockIdx.x * TB + t;
  const bool live = q < nsample;
  float* grad = rows + (size_t)(blockIdx.x >> 1) * kTrainRow;
  float f[NF];
  float ytrue = 0.0f;
  if (live) {
    long long g;
    if (idx) {
      g = idx[q];
    } else {  // a random system and a random entry among those the network predicts
      const uint64_t h = mix64(seed ^ (0x9E3779B97F4A7C15ull * (uint64_t)(q + 1)));
      g = (long long)(h % (uint64_t)nsys) * P.nnz + P.mlp_ent[(h >> 32) % (uint64_t)P.n_mlp];
    }
    const int s = (int)(g / P.nnz), e = (int)(g % P.nnz);
    const Feat ft = features(P, s, e, A, rown, coln, corr);
#pragma unroll
    for (int k = 0; k < NF; ++k) f[k] = ft.f[k];
    const double denom = ft.a * (double)ft.base;
    ytrue = denom != 0.0 ? (float)(LUt[g] / denom - 1.0) : 0.0f;
  } else {
#pragma unroll
    for (int k = 0; k < NF; ++k) f[k] = 0.0f;
  }
#pragma unroll
  for (int k = 0; k < NF; ++k) X[t * NF + k] = live ? f[k] : 0.0f;
  // ---- layer 1 (CUDA cores): H1 hi / lo into A1 (row t) and BT (column t), gelu'(pre1) into G1
  __nv_bfloat16* bth = reinterpret_cast<__nv_bfloat16*>(smt + TR_BT);
  __nv_bfloat16* btl = reinterpret_cast<__nv_bfloat16*>(smt + TR_BT + H * TB * 2);
#pragma unroll 1
  for (int c = 0; c < H / 8; ++c) {
    __align__(16) __nv_bfloat16 hi[8], lo[8];
#pragma unroll
    for (int d = 0; d < 8; ++d) {
      const int v = 8 * c + d;
      const float4 wa = w1v[v * 3], wb = w1v[v * 3 + 1], wc = w1v[v * 3 + 2];
      const float w[NF] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w, wc.x};
      float pre = wc.y;
#pragma unroll
      for (int k = 0; k < NF; ++k) pre = fmaf(w[k], f[k], pre);
      const float h = live ? gelu(pre) : 0.0f;
      G1[t * LD + v] = live ? gelu_d(pre) : 0.0f;
      split_bf16(h, hi[d], lo[d]);
      const uint32_t bo = tc::kmajor_off(v, t, TB) / 2;
      bth[bo] = hi[d];
      btl[bo] = lo[d];
    }
    const uint32_t off = tc::kmajor_off(t, 8 * c, H);
    *reinterpret_cast<uint4*>(smt + TR_A1 + off) = *reinterpret_cast<const uint4*>(hi);
    *reinterpret_cast<uint4*>(smt + TR_A1 + TB * H * 2 + off) = *reinterpret_cast<const uint4*>(lo);
  }
  const uint32_t a1h = tc::smem_u32(smt + TR_A1), a1l = a1h + TB * H * 2;
  const uint32_t bth_a = tc::smem_u32(smt + TR_BT), btl_a = bth_a + H * TB * 2;
  const uint32_t at_a = tc::smem_u32(smt + TR_AT), bw_a = tc::smem_u32(smt + TR_BW), bwt_a = tc::smem_u32(smt + TR_BWT);
  constexpr uint32_t kSbo64 = H * 16, kSbo128 = TB * 16;
  const uint32_t id128 = tc::idesc_bf16(128, H);
  // ---- forward layer 2 on the tensor cores: D1 = H1 W2^T
  tc::fence_smem_to_async();
  tc::fence_before_sync();
  __syncthreads();
  if (t == 0) {
    tc::fence_after_sync();
#pragma unroll
    for (int j = 0; j < H / 16; ++j)
      tc::mma_bf16(tmem, tc::sdesc(a1h + 256 * j, kSbo64), tc::sdesc(bw_a + 256 * j, kSbo64), id128, j > 0);
#pragma unroll
    for (int j = 0; j < H / 16; ++j)
      tc::mma_bf16(tmem, tc::sdesc(a1l + 256 * j, kSbo64), tc::sdesc(bw_a + 256 * j, kSbo64), id128, 1);
    tc::commit(&s_mbar);
  }
  if (!tc::mbar_wait(&s_mbar, 0, kWaitLimit)) s_fail = 1;  // 1 + the parity of the phase that did not complete
  tc::fence_after_sync();
  __syncthreads();
  if (!s_fail) {
    // ---- output layer, loss, dout
    float out = b3;
#pragma unroll 1
    for (int c = 0; c < H / 16; ++c) {
      float acc[16];
      tc::ld16(trow + 16 * c, acc);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const float2 bw = bwv[16 * c + k];
        out = fmaf(bw.y, gelu(acc[k] + bw.x), out);
      }
    }
    const float diff = out - ytrue;
    const float err2 = live ? diff * diff : 0.0f;
    const float dout = live ? 2.0f * diff * scale : 0.0f;
    // ---- dpre2 = dout w3 gelu'(pre2) into A1 (row t) and AT (column t); per-unit sums of dpre2 (db2)
    // and of dout gelu(pre2) (dW3), reduce-scattered over the warp: lane l holds units l and 32 + l
    __nv_bfloat16* ath = reinterpret_cast<__nv_bfloat16*>(smt + TR_AT);
    float rs_db2[2], rs_dw3[2];
#pragma unroll 1
    for (int c2 = 0; c2 < 2; ++c2) {
      float dp[32], dw[32];
#pragma unroll
      for (int h16 = 0; h16 < 2; ++h16) {
        float acc[16];
        tc::ld16(trow + 32 * c2 + 16 * h16, acc);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const int u = 32 * c2 + 16 * h16 + k;
          const float pre = acc[k] + bwv[u].x;
          dp[16 * h16 + k] = dout * bwv[u].y * gelu_d(pre);
          dw[16 * h16 + k] = dout * gelu(pre);
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        __align__(16) __nv_bfloat16 hi[8], lo[8];
#pragma unroll
        for (int d = 0; d < 8; ++d) {
          const int u = 32 * c2 + 8 * c + d;
          split_bf16(dp[8 * c + d], hi[d], lo[d]);
          ath[tc::kmajor_off(u, t, TB) / 2] = hi[d];
          ath[tc::kmajor_off(H + u, t, TB) / 2] = lo[d];
        }
        const uint32_t off = tc::kmajor_off(t, 32 * c2 + 8 * c, H);
        *reinterpret_cast<uint4*>(smt + TR_A1 + off) = *reinterpret_cast<const uint4*>(hi);
        *reinterpret_cast<uint4*>(smt + TR_A1 + TB * H * 2 + off) = *reinterpret_cast<const uint4*>(lo);
      }
      rs_db2[c2] = warp_reduce_scatter32(dp);
      rs_dw3[c2] = warp_reduce_scatter32(dw);
    }
    // ---- backward GEMMs on the tensor cores: D2 = dpre2 W2, D3 / D4 = dpre2^T (hi | lo stacked) H1 (hi / lo)
    tc::fence_smem_to_async();
    tc::fence_before_sync();
    __syncthreads();
    if (t == 0) {
      tc::fence_after_sync();
#pragma unroll
      for (int j = 0; j < H / 16; ++j)
        tc::mma_bf16(tmem + 64, tc::sdesc(a1h + 256 * j, kSbo64), tc::sdesc(bwt_a + 256 * j, kSbo64), id128, j > 0);
#pragma unroll
      for (int j = 0; j < H / 16; ++j)
        tc::mma_bf16(tmem + 64, tc::sdesc(a1l + 256 * j, kSbo64), tc::sdesc(bwt_a + 256 * j, kSbo64), id128, 1);
#pragma unroll
      for (int j = 0; j < TB / 16; ++j)
        tc::mma_bf16(tmem + 128, tc::sdesc(at_a + 256 * j, kSbo128), tc::sdesc(bth_a + 256 * j, kSbo128), id128,
                     j > 0);
#pragma unroll
      for (int j = 0; j < TB / 16; ++j)
        tc::mma_bf16(tmem + 192, tc::sdesc(at_a + 256 * j, kSbo128), tc::sdesc(btl_a + 256 * j, kSbo128), id128,
                     j > 0);
      tc::commit(&s_mbar);
    }
    // loss and the sum of dout (db3) while the tensor cores run
    float l = err2, dsum = dout;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      l += __shfl_down_sync(kFull, l, off);
      dsum += __shfl_down_sync(kFull, dsum, off);
    }
    if (lane == 0) {
      s_loss[warp] = l;
      s_do[warp] = dsum;
    }
    RED[(0 * 4 + warp) * H + lane] = rs_db2[0];
    RED[(0 * 4 + warp) * H + 32 + lane] = rs_db2[1];
    RED[(1 * 4 + warp) * H + lane] = rs_dw3[0];
    RED[(1 * 4 + warp) * H + 32 + lane] = rs_dw3[1];
    if (!tc::mbar_wait(&s_mbar, 1, kWaitLimit)) s_fail = 2;
    tc::fence_after_sync();
    __syncthreads();
    if (!s_fail) {
      // ---- dpre1 = dh1 * gelu'(pre1) into G1; per-unit sums of dpre1 (db1)
      float rs_db1[2];
#pragma unroll 1
      for (int c2 = 0; c2 < 2; ++c2) {
        float dp[32];
#pragma unroll
        for (int h16 = 0; h16 < 2; ++h16) {
          float acc[16];
          tc::ld16(trow + 64 + 32 * c2 + 16 * h16, acc);
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const int v = 32 * c2 + 16 * h16 + k;
            const float d = acc[k] * G1[t * LD + v];
            G1[t * LD + v] = d;
            dp[16 * h16 + k] = d;
          }
        }
        rs_db1[c2] = warp_reduce_scatter32(dp);
      }
      RED[(2 * 4 + warp) * H + lane] = rs_db1[0];
      RED[(2 * 4 + warp) * H + 32 + lane] = rs_db1[1];
      // ---- dW2: row r of D3 + D4 is unit r % 64's share (high part for r < 64, low part above); the low
      // parts go through shared memory (AT's, which the tensor cores have read)
      float* W2L = reinterpret_cast<float*>(smt + TR_AT) + (t & 63) * LD;
      auto dw2 = [&](auto put) {
#pragma unroll 1
        for (int c = 0; c < H / 16; ++c) {
          float d3[16], d4[16];
          tc::ld16(trow + 128 + 16 * c, d3);
          tc::ld16(trow + 192 + 16 * c, d4);
          put(16 * c, d3, d4);
        }
      };
      if (warp >= 2)
        dw2([&](int o, const float(&d3)[16], const float(&d4)[16]) {
#pragma unroll
          for (int k = 0; k < 16; ++k) W2L[o + k] = d3[k] + d4[k];
        });
      __syncthreads();
      if (warp < 2)
        dw2([&](int o, const float(&d3)[16], const float(&d4)[16]) {
#pragma unroll
          for (int k = 0; k < 16; k += 4)
            atomicAdd(reinterpret_cast<float4*>(grad + OW2 + t * H + o + k),
                      make_float4((d3[k] + d4[k]) + W2L[o + k], (d3[k + 1] + d4[k + 1]) + W2L[o + k + 1],
                                  (d3[k + 2] + d4[k + 2]) + W2L[o + k + 2], (d3[k + 3] + d4[k + 3]) + W2L[o + k + 3]));
        });
      if (t == 0) {
        float a = 0.0f, d = 0.0f;
        for (int w = 0; w < TB / 32; ++w) {
          a += s_loss[w];
          d += s_do[w];
        }
        atomicAdd(grad + kMlpParams, a * scale);
        atomicAdd(grad + OB3, d);
      }
      if (t < H) {
        float db2 = 0.0f, dw3 = 0.0f, db1 = 0.0f;
        for (int w = 0; w < TB / 32; ++w) {
          db2 += RED[(0 * 4 + w) * H + t];
          dw3 += RED[(1 * 4 + w) * H + t];
          db1 += RED[(2 * 4 + w) * H + t];
        }
        atomicAdd(grad + OB2 + t, db2);
        atomicAdd(grad + OW3 + t, dw3);
        atomicAdd(grad + OB1 + t, db1);
      }
      for (int k = t; k < H * NF; k += TB) {  // dW1[u][f] = sum_t dpre1[t][u] * x[t][f]
        const int u = k / NF, fi = k % NF;
        float acc = 0.0f;
        for (int r = 0; r < TB; ++r) acc = fmaf(G1[r * LD + u], X[r * NF + fi], acc);
        atomicAdd(grad + OW1 + k, acc);
      }
    }
  }
  if (s_fail && t == 0) atomicAdd(grad + kMlpParams, __int_as_float(0x7fc00000));
  // a round that timed out may still be in flight: wait once more (bounded) before freeing its columns
  if (s_fail) tc::mbar_wait(&s_mbar, (uint32_t)(s_fail - 1), kWaitLimit);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::dealloc(tmem, kTrainTmemCols);
}

// The gradient and the loss from the blocks' rows, in an order that only the
// number of rows sets: warp w of a CTA adds rows w, w + 16, ... of 32 columns,
// one column per lane, then the first warp adds the 16 sums.  Every addition
// keeps its rounding error (Knuth's two-sum), so the result is the sum's
// correctly rounded value but for a few ulps of the errors' own sum: nearer to
// it than any order of plain additions.  acc / cor: the sum and its error so
// far, continued over the parts of a large batch (start: its first part).
// Leaves the rows zero for the next part.
// Reads 19.5 KB per row: 256 rows (65536 samples) about 3 us.
constexpr int kSumWarps = 16;
__device__ __forceinline__ void two_sum(float& s, float& c, float x) {
  const float t = s + x, z = t - s;
  c += (s - (t - z)) + (x - z);
  s = t;
}
__global__ void __launch_bounds__(32 * kSumWarps) k_grad_sum(float* rows, int nrows, int start,
                                                            float* __restrict__ acc, float* __restrict__ cor,
                                                            float* __restrict__ grad, float* __restrict__ loss) {
  __shared__ float s_s[kSumWarps][32], s_c[kSumWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
  float s = 0.0f, c = 0.0f;
  if (k <= kMlpParams) {
    for (int r = warp; r < nrows; r += 8 * kSumWarps) {
      float x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = r + j * kSumWarps < nrows ? rows[(size_t)(r + j * kSumWarps) * kTrainRow + k] : 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        two_sum(s, c, x[j]);
        if (r + j * kSumWarps < nrows) rows[(size_t)(r + j * kSumWarps) * kTrainRow + k] = 0.0f;
      }
    }
  }
  s_s[warp][lane] = s;
  s_c[warp][lane] = c;
  __syncthreads();
  if (warp != 0 || k > kMlpParams) return;
  s = start ? 0.0f : acc[k];
  c = start ? 0.0f : cor[k];
  for (int w = 0; w < kSumWarps; ++w) {
    two_sum(s, c, s_s[w][lane]);
    c += s_c[w][lane];
  }
  acc[k] = s;
  cor[k] = c;
  const float v = isfinite(s) ? s + c : s;  // the error of an infinite sum is NaN
  if (k < kMlpParams)
    grad[k] = v;
  else
    *loss = v;
}

// Adam on the FP32 master parameters; refreshes the BF16 copy.
__global__ void k_adam(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ g, __nv_bfloat16* __restrict__ pbf, int count, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const float gk = g[k];
  const float mk = b1 * m[k] + (1.0f - b1) * gk;
  const float vk = b2 * v[k] + (1.0f - b2) * gk * gk;
  m[k] = mk;
  v[k] = vk;
  const float pk = p[k] - lr * (mk / c1) / (sqrtf(vk / c2) + eps);
  p[k] = pk;
  pbf[k] = __float2bfloat16_rn(pk);
}

__global__ void k_to_bf16(const float* __restrict__ p, __nv_bfloat16* __restrict__ pbf, int count) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) pbf[k] = __float2bfloat16_rn(p[k]);
}

// Features and forward outputs of given samples (checks against the oracle).
__global__ void k_mlp_eval(const DevPattern P, int nsys, const double* __restrict__ A, const float* __restrict__ rown,
                           const float* __restrict__ coln, const float* __restrict__ corr,
                           const __nv_bfloat16* __restrict__ pbf, int nsample, const int* __restrict__ idx,
                           float* __restrict__ feat, float* __restrict__ out, double* __restrict__ base) {
  extern __shared__ __align__(16) float sm[];
  stage_params(pbf, sm);
  __syncthreads();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nsample) return;
  const long long g = idx[q];
  const Feat ft = features(P, (int)(g / P.nnz), (int)(g % P.nnz), A, rown, coln, corr);
  for (int k = 0; k < NF; ++k) feat[(size_t)q * NF + k] = ft.f[k];
  base[q] = ft.base;
  out[q] = mlp_forward(sm, ft.f, nullptr, nullptr, nullptr);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo_elem, float hi_elem) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo_elem, hi_elem);  // .x = first (low 16 bits)
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Warm start: persistent CTAs of 128 threads over the systems (the network's
// weights are staged once per CTA).  Every system's LU0 starts as a copy of A
// (exact for the entries on or above the diagonal without dependency pairs,
// which converge to a_ij).  The other entries go through the network in tiles
// of 128, one entry per thread, both hidden layers on the tensor core
// (tcgen05.mma, M = 128 entries, N = 64, BF16 operands split into high and low
// parts so that x = hi + lo to about 16 bits, FP32 accumulation in the same 64
// TMEM columns), issued by one thread and completed through an mbarrier:
//   layer 1: the features (9, then 1.0 for the bias, zero-padded to K = 16)
//   against W1 | b1 (BF16): 2 MMAs;
//   every thread reads its row of pre1 (tcgen05.ld, lane = row), GELU, and
//   stores the activations as the 128 x 64 A operands of layer 2;
//   layer 2: hi and lo against W2 (BF16), K = 64: 8 MMAs; while they run,
//   every thread gathers the features of its entry of the next tile;
//   every thread reads its row of pre2, adds b2, GELU, the output layer's dot
//   product with w3, and writes its prediction into LU0.
// The ILU residual ||(A - L0 U0)|_S||_F / ||A||_F of the written factors then
// decides between the prediction and the plain initialisation (the predicted
// entries are copied back from A).  Shared memory holds only the operands and
// weights (42.5 KB; the layer-1 operand lives in the layer-2 low-part buffer,
// which is free until layer 1 has completed), so five CTAs share an SM.
// The mbarrier waits are bounded: a CTA whose tensor-core work does not
// complete in time stops using it and writes the plain initialisation
// (used = 0, ILU residual -1) for its remaining systems.
constexpr int WARM_THREADS = 128;
constexpr int KX = 16;  // layer-1 K: 9 features, the bias input, zero padding
constexpr int WT_AH = 0, WT_AL = WT_AH + 128 * H * 2, WT_B = WT_AL + 128 * H * 2, WT_B1 = WT_B + H * H * 2;
constexpr int WT_BW = WT_B1 + H * KX * 2, WT_SMEM = WT_BW + H * 8;
constexpr int WT_XH = WT_AL, WT_XL = WT_AL + 128 * KX * 2;  // layer-1 operand, aliasing the layer-2 low part
constexpr uint32_t kTmemCols = 64;
static_assert(WT_B1 % 16 == 0 && WT_BW % 16 == 0 && WT_XL + 128 * KX * 2 <= WT_B, "aligned operand blocks");

// features of predicted entry q of system s (zeros past the last one)
__device__ __forceinline__ void warm_features(const DevPattern& P, int s, int q, const double* __restrict__ A,
                                              const float* __restrict__ rown, const float* __restrict__ coln,
                                              const float* __restrict__ corr, float (&f)[NF], double& ab, int& e) {
  if (q < P.n_mlp) {
    e = P.mlp_ent[q];
    const Feat ft = features(P, s, e, A, rown, coln, corr);
#pragma unroll
    for (int k = 0; k < NF; ++k) f[k] = ft.f[k];
    ab = ft.a * (double)ft.base;
  } else {
    e = -1;
    ab = 0.0;
#pragma unroll
    for (int k = 0; k < NF; ++k) f[k] = 0.0f;
  }
}

__global__ void __launch_bounds__(WARM_THREADS) k_mlp_warm(const DevPattern P, int nsys,
                                                           const double* __restrict__ A,
                                                           const float* __restrict__ rown,
                                                           const float* __restrict__ coln,
                                                           const float* __restrict__ corr,
                                                           const __nv_bfloat16* __restrict__ pbf, double threshold,
                                                           double* __restrict__ LU0, double* __restrict__ res_out,
                                                           int* __restrict__ used) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  __shared__ uint64_t s_mbar;
  __shared__ uint32_t s_tmem;
  __shared__ double s_num[WARM_THREADS / 32], s_den[WARM_THREADS / 32];
  __shared__ int s_ok, s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // weights: W2 as the K-major B operand of layer 2 (row u = output unit, k = input unit), W1 | b1 as the
  // K-major B operand of layer 1 (row v: W1[v][0..8], b1[v], zeros), (b2, w3) pairs
  {
    const uint4* w2g = reinterpret_cast<const uint4*>(pbf + OW2);  // row u: 8 chunks of 8 BF16
    for (int k = tid; k < H * 8; k += WARM_THREADS) {
      const int u = k >> 3, c = k & 7;
      *reinterpret_cast<uint4*>(smraw + WT_B + tc::kmajor_off(u, 8 * c, H)) = w2g[k];
    }
    for (int k = tid; k < H * KX; k += WARM_THREADS) {
      const int v = k / KX, c = k % KX;
      const __nv_bfloat16 w = c < NF ? pbf[OW1 + v * NF + c] : (c == NF ? pbf[OB1 + v] : __float2bfloat16_rn(0.0f));
      *reinterpret_cast<__nv_bfloat16*>(smraw + WT_B1 + tc::kmajor_off(v, c, KX)) = w;
    }
    float2* bw = reinterpret_cast<float2*>(smraw + WT_BW);
    for (int u = tid; u < H; u += WARM_THREADS) bw[u] = make_float2(__bfloat162float(pbf[OB2 + u]), __bfloat162float(pbf[OW3 + u]));
  }
  if (tid == 0) {
    tc::mbar_init(&s_mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_fail = 0;
  }
  if (warp == 0) tc::alloc(&s_tmem, kTmemCols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = s_tmem;
  const float2* bw = reinterpret_cast<const float2*>(smraw + WT_BW);
  const float b3 = __bfloat162float(pbf[OB3]);
  const uint32_t a_hi = tc::smem_u32(smraw + WT_AH), a_lo = tc::smem_u32(smraw + WT_AL);
  const uint32_t x_hi = tc::smem_u32(smraw + WT_XH), x_lo = tc::smem_u32(smraw + WT_XL);
  const uint32_t b_w2 = tc::smem_u32(smraw + WT_B), b_w1 = tc::smem_u32(smraw + WT_B1);
  constexpr uint32_t kSbo = H * 16, kSboX = KX * 16;  // 8-row groups 1024 / 256 bytes apart
  const uint32_t idesc = tc::idesc_bf16(128, H);
  const uint32_t trow = tmem + ((uint32_t)(32 * warp) << 16);  // this warp's 32 TMEM lanes
  const int ntile = (P.n_mlp + WARM_THREADS - 1) / WARM_THREADS;
  uint32_t phase = 0;
  // one tensor-core round: wait (bounded) for the MMAs committed last, then make the accumulator readable;
  // false (uniformly) when the round did not complete
  auto round_done = [&]() {
    const bool done = tc::mbar_wait(&s_mbar, phase, kWaitLimit);
    phase ^= 1u;
    if (!done) s_fail = 1;
    tc::fence_after_sync();
    __syncthreads();
    return s_fail == 0;
  };
  for (int s = blockIdx.x; s < nsys; s += gridDim.x) {
    const double* As = A + (size_t)s * P.nnz;
    double* Ls = LU0 + (size_t)s * P.nnz;
    for (int e = tid; e < P.nnz; e += WARM_THREADS) Ls[e] = As[e];
    const bool failed = s_fail != 0;  // uniform: written before the last barrier
    float f[NF];
    double ab = 0.0;
    int e = -1;
    if (!failed) warm_features(P, s, tid, A, rown, coln, corr, f, ab, e);
    __syncthreads();  // the copy of A is complete before any prediction overwrites it
    for (int tile = 0; tile < ntile && !failed; ++tile) {
      // ---- layer 1: this entry's features (and 1.0 for the bias) as row tid of the K = 16 operand
      {
        __align__(16) __nv_bfloat16 hi[KX], lo[KX];
#pragma unroll
        for (int k = 0; k < KX; ++k) {
          const float x = k < NF ? f[k] : (k == NF ? 1.0f : 0.0f);
          hi[k] = __float2bfloat16_rn(x);
          lo[k] = __float2bfloat16_rn(x - __bfloat162float(hi[k]));
        }
#pragma unroll
        for (int c = 0; c < KX / 8; ++c) {
          const uint32_t off = tc::kmajor_off(tid, 8 * c, KX);
          *reinterpret_cast<uint4*>(smraw + WT_XH + off) = reinterpret_cast<const uint4*>(hi)[c];
          *reinterpret_cast<uint4*>(smraw + WT_XL + off) = reinterpret_cast<const uint4*>(lo)[c];
        }
      }
      tc::fence_smem_to_async();
      tc::fence_before_sync();  // every thread's previous accumulator reads are done
      __syncthreads();
      if (tid == 0) {
        tc::fence_after_sync();
        tc::mma_bf16(tmem, tc::sdesc(x_hi, kSboX), tc::sdesc(b_w1, kSboX), idesc, 0);
        tc::mma_bf16(tmem, tc::sdesc(x_lo, kSboX), tc::sdesc(b_w1, kSboX), idesc, 1);
        tc::commit(&s_mbar);
      }
      if (!round_done()) break;
      // ---- GELU of this row of pre1 into the layer-2 operands (hi and lo), 16 units at a time
#pragma unroll 1
      for (int c = 0; c < H / 16; ++c) {
        float acc[16];
        tc::ld16(trow + 16 * c, acc);
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int d = 0; d < 16; d += 2) {
          const float h0 = gelu_fast(acc[d]), h1 = gelu_fast(acc[d + 1]);
          const float g0 = __bfloat162float(__float2bfloat16_rn(h0));
          const float g1 = __bfloat162float(__float2bfloat16_rn(h1));
          hi[d >> 1] = pack_bf16(g0, g1);
          lo[d >> 1] = pack_bf16(h0 - g0, h1 - g1);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint32_t off = tc::kmajor_off(tid, 16 * c + 8 * q, H);
          *reinterpret_cast<uint4*>(smraw + WT_AH + off) = make_uint4(hi[4 * q], hi[4 * q + 1], hi[4 * q + 2], hi[4 * q + 3]);
          *reinterpret_cast<uint4*>(smraw + WT_AL + off) = make_uint4(lo[4 * q], lo[4 * q + 1], lo[4 * q + 2], lo[4 * q + 3]);
        }
      }
      // ---- layer 2
      tc::fence_smem_to_async();
      tc::fence_before_sync();
      __syncthreads();
      if (tid == 0) {
        tc::fence_after_sync();
#pragma unroll
        for (int j = 0; j < H / 16; ++j)
          tc::mma_bf16(tmem, tc::sdesc(a_hi + 256 * j, kSbo), tc::sdesc(b_w2 + 256 * j, kSbo), idesc, j > 0);
#pragma unroll
        for (int j = 0; j < H / 16; ++j)
          tc::mma_bf16(tmem, tc::sdesc(a_lo + 256 * j, kSbo), tc::sdesc(b_w2 + 256 * j, kSbo), idesc, 1);
        tc::commit(&s_mbar);
      }
      // the next tile's features while the tensor core runs
      const double ab_cur = ab;
      const int e_cur = e;
      if (tile + 1 < ntile) warm_features(P, s, (tile + 1) * WARM_THREADS + tid, A, rown, coln, corr, f, ab, e);
      if (!round_done()) break;
      // ---- this thread's row of pre2: b2, GELU, output layer
      float out = 0.0f;
#pragma unroll 1
      for (int c = 0; c < H / 16; ++c) {
        float acc[16];
        tc::ld16(trow + 16 * c, acc);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float2 q2 = bw[16 * c + k];
          out = fmaf(q2.y, gelu_fast(acc[k] + q2.x), out);
        }
      }
      if (e_cur >= 0) Ls[e_cur] = ab_cur * (1.0 + (double)(out + b3));
      tc::fence_before_sync();
    }
    __syncthreads();  // every prediction of this system written (block-visible) before the residual reads
    const bool fail = s_fail != 0;
    // residual of the warm start: (A - LU)_ij = a_ij - sum_{k<min(i,j)} l_ik u_kj - (l_ij u_jj | u_ij)
    double num = 0.0, den = 0.0;
    if (!fail) {
      for (int e2 = tid; e2 < P.nnz; e2 += WARM_THREADS) {
        const int i = P.row_of[e2], j = P.ci[e2];
        double acc = 0.0;
        for (int q = P.dep_ptr[e2]; q < P.dep_ptr[e2 + 1]; ++q) {
          const int2 d = P.dep[q];
          acc = fma(Ls[d.x], Ls[d.y], acc);
        }
        acc = (j < i) ? fma(Ls[e2], Ls[P.diag[j]], acc) : acc + Ls[e2];
        const double rr = As[e2] - acc;
        num = fma(rr, rr, num);
        den = fma(As[e2], As[e2], den);
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      num += __shfl_down_sync(kFull, num, off);
      den += __shfl_down_sync(kFull, den, off);
    }
    if (lane == 0) {
      s_num[warp] = num;
      s_den[warp] = den;
    }
    __syncthreads();
    if (tid == 0) {
      double a = 0.0, b = 0.0;
      for (int w = 0; w < WARM_THREADS / 32; ++w) {
        a += s_num[w];
        b += s_den[w];
      }
      const double res = fail ? -1.0 : (b > 0.0 ? sqrt(a / b) : sqrt(a));
      s_ok = (!fail && res <= threshold) ? 1 : 0;  // NaN fails the test: fallback
      if (res_out) res_out[s] = res;
      if (used) used[s] = s_ok;
    }
    __syncthreads();
    if (!s_ok) {  // fallback: the predicted entries back to A's values
      for (int q = tid; q < P.n_mlp; q += WARM_THREADS) {
        const int e2 = P.mlp_ent[q];
        Ls[e2] = As[e2];
      }
    }
    __syncthreads();  // s_ok and the residual slots are free for the next system
  }
  // a tensor-core round that timed out may still be in flight: wait for it once more (bounded) before the
  // accumulator columns are freed
  if (s_fail) tc::mbar_wait(&s_mbar, phase ^ 1u, kWaitLimit);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::dealloc(tmem, kTmemCols);
}

}  // namespace

cudaError_t launch_mlp_rowstats(const DevPattern& p, int nsys, const double* A, float* rown, float* coln, float* corr,
                                cudaStream_t st) {
  if (nsys == 0) return cudaSuccess;
  k_rowstats<<<nsys, 256, 0, st>>>(p, nsys, A, rown, coln, corr);
  return cudaGetLastError();
}

size_t mlp_train_smem() { return TR_SMEM; }

cudaError_t launch_mlp_train(const DevPattern& p, int nsys, const double* A, const double* LUt, const float* rown,
                             const float* coln, const float* corr, const void* pbf, int nsample, const int* idx,
                             uint64_t seed, float* work, int nrows, float* grad, float* loss, cudaStream_t st) {
  if (nsample == 0) return cudaSuccess;
  const size_t smem = mlp_train_smem();
  cudaError_t e = cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  float *acc = work, *cor = work + kTrainRow, *rows = work + 2 * kTrainRow;
  const long long blocks = ((long long)nsample + TB - 1) / TB;
  for (long long b = 0; b < blocks; b += 2LL * nrows) {
    const int part = (int)std::min<long long>(2LL * nrows, blocks - b), used = (part + 1) / 2;
    k_mlp_train<<<part, TB, smem, st>>>(p, nsys, A, LUt, rown, coln, corr, (const __nv_bfloat16*)pbf, nsample, idx,
                                        seed, 1.0f / (float)nsample, b * TB, rows);
    k_grad_sum<<<(kMlpParams + 32) / 32, 32 * kSumWarps, 0, st>>>(rows, used, b == 0, acc, cor, grad, loss);
  }
  return cudaGetLastError();
}

// Rows of the gradient parts kept at a time: one per two blocks, at most four per SM (12 MB), whole waves of the
// training kernel's one CTA per SM.
int mlp_train_rows(int nsample, int nsm) {
  return (int)std::min(((long long)nsample + 2 * TB - 1) / (2 * TB), 4LL * nsm);
}
size_t mlp_train_work(int nrows) { return (size_t)(nrows + 2) * kTrainRow * sizeof(float); }

cudaError_t launch_mlp_adam(float* p, float* m, float* v, const float* g, void* pbf, int count, float lr, int step,
                            cudaStream_t st) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  k_adam<<<(count + 255) / 256, 256, 0, st>>>(p, m, v, g, (__nv_bfloat16*)pbf, count, lr, b1, b2, eps, c1, c2);
  return cudaGetLastError();
}

cudaError_t launch_mlp_to_bf16(const float* p, void* pbf, int count, cudaStream_t st) {
  k_to_bf16<<<(count + 255) / 256, 256, 0, st>>>(p, (__nv_bfloat16*)pbf, count);
  return cudaGetLastError();
}

cudaError_t launch_mlp_eval(const DevPattern& p, int nsys, const double* A, const float* rown, const float* coln,
                            const float* corr, const void* pbf, int nsample, const int* idx, float* feat, float* out,
                            double* base, cudaStream_t st) {
  if (nsample == 0) return cudaSuccess;
  const size_t smem = sizeof(float) * ((kMlpParams + 3) & ~3);
  k_mlp_eval<<<(nsample + 127) / 128, 128, smem, st>>>(p, nsys, A, rown, coln, corr, (const __nv_bfloat16*)pbf,
                                                       nsample, idx, feat, out, base);
  return cudaGetLastError();
}

cudaError_t launch_mlp_warm(const DevPattern& p, int nsys, const double* A, const float* rown, const float* coln,
                            const float* corr, const void* pbf, double threshold, double* lu0, double* res, int* used,
                            cudaStream_t st) {
  if (nsys == 0) return cudaSuccess;
  const size_t smem = WT_SMEM;
  cudaError_t e = cudaFuncSetAttribute(k_mlp_warm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // CTAs per SM from the kernel's own resources (measured on GB300: the occupancy calculator reports
  // one CTA per SM for this tcgen05 kernel, where its shared memory admits five); every resident CTA
  // holds kTmemCols of the SM's 512 TMEM columns, so at most 512 / kTmemCols, and no allocation ever
  // waits for another CTA's
  int dev = 0, nsm = 0, per_sm = 0, reserved = 0, thr_sm = 0, regs_sm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  cudaDeviceGetAttribute(&thr_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev);
  cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev);
  cudaFuncAttributes fa;
  e = cudaFuncGetAttributes(&fa, k_mlp_warm);
  if (e != cudaSuccess) return e;
  int occ = per_sm / (int)(smem + fa.sharedSizeBytes + reserved);
  occ = std::min(occ, thr_sm / WARM_THREADS);
  occ = std::min(occ, regs_sm / std::max(1, ((fa.numRegs + 7) / 8 * 8) * WARM_THREADS));
  occ = std::max(1, std::min(occ, 512 / (int)kTmemCols));
  const int grid = nsys < nsm * occ ? nsys : nsm * occ;
  k_mlp_warm<<<grid, WARM_THREADS, smem, st>>>(p, nsys, A, rown, coln, corr, (const __nv_bfloat16*)pbf, threshold,
                                               lu0, res, used);
  return cudaGetLastError();
}

}  // namespace bilu
