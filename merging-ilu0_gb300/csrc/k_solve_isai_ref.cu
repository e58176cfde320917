// Reference-order BiCGSTAB with the ISAI of L and U (PrecondBiCGSTAB_ilu_isai_gpu.cu:89-257):
// several systems of a batch per CTA, in step.
//
// The reference sums the inner products of this solver serially
// (Bicgstab_common.hpp:82-95), one FMA after another over the rows, and every
// iterate depends on their bits.  With one CTA per system (k_solve.cu) each such
// sum is a warp instruction per row with one lane active, and on GB300 an FP64
// instruction costs the same with one lane as with 32: at 16x16 the six sums of
// an iteration were 1536 of its 2417 FP64 instructions, on a pipe 78 % busy.
// Here lane g of the first warp runs the chain of system g, so one instruction
// serves every system of the CTA, and the scalar recurrences of all of them are
// formed by the same lanes.  The pairs of sums that do not depend on each other
// ((t,s) and (t,t); (r,r) and the next (r,r_hat)) run on the two half-warps.
// Vectors x, r, p, v, t are in registers (R rows per thread); shared memory
// holds what other threads read: p / p_hat, r / s, the ISAI intermediate / v / t
// and r_hat.  Two CTAs per SM, so that one's chains (64 clocks per term) overlap
// the other's SpMVs.  Row trees have the slots of the stencils' own row lengths
// (row_ref).  A system that has stopped waits for the others of its CTA.
// Same operations per system in the same order as k_bicgstab<FT, true>, so the
// same bits.  Measured: ILU(0)-ISAI solve of 2048 2D 16x16
// systems 4.20 -> 1.74 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "bilu_internal.h"

namespace bilu {
namespace {

constexpr unsigned kFull = 0xffffffffu;

#include "k_row_ref.cuh"

constexpr int kThreads = 256, kMaxSys = 8;  // per CTA

struct IsaiRefArgs {
  SolveArgs s;
  int per_cta;  // systems per CTA
  int tsys;     // threads per system (whole warps)
  int stride;   // doubles per system in shared memory, odd: lanes of different systems read different banks
};

// y = row i of M x in the reference's tree (MI = longest row, S its power of two)
template <int S, int M, typename IT>
__device__ __forceinline__ double tree(const double* __restrict__ a, const IT* __restrict__ ci,
                                       const int* __restrict__ rp, int i, const double* x) {
  const int beg = __ldg(rp + i);
  return row_ref<S, M>(a, ci, beg, __ldg(rp + i + 1) - beg, x);
}

__device__ __forceinline__ float row_seq(const float* __restrict__ a, const unsigned short* __restrict__ ci,
                                         const int* __restrict__ rp, int i, const float* x) {
  float acc = 0.0f;
  const int e = __ldg(rp + i + 1);
  for (int k = __ldg(rp + i); k < e; ++k) acc = fmaf(a[k], x[__ldg(ci + k)], acc);
  return acc;
}

// sum of fma(a_i, b_i, .) over i = 0 .. n-1 in order, from 0
__device__ __forceinline__ double chain(const double* a, const double* b, int n) {
  double acc = 0.0;
  int i = 0;
  for (; i + 8 <= n; i += 8) {
    double u[8], w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      u[j] = a[i + j];
      w[j] = b[i + j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) acc = fma(u[j], w[j], acc);
  }
  for (; i < n; ++i) acc = fma(a[i], b[i], acc);
  return acc;
}

// SA, MA / SI, MI: row trees of A and of the FP64 ISAI values
template <int R, typename FT, int SA, int MA, int SI, int MI>
__global__ void __launch_bounds__(kThreads, 2) k_bicgstab_isai_ref(const IsaiRefArgs u) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double s_a[kMaxSys], s_b[kMaxSys];  // the scalars a step broadcasts
  __shared__ int s_on[kMaxSys], s_any;           // systems still iterating
  const SolveArgs& a = u.s;
  const DevPattern& P = a.pat;
  constexpr bool kFP32 = sizeof(FT) == 4;
  const int n = P.n, tid = threadIdx.x, lane = tid & 31, ts = u.tsys;
  const int g = tid / ts, t0 = tid - g * ts;  // system of the CTA, thread of the system
  const int sys = blockIdx.x * u.per_cta + g;
  const int nsys = min(u.per_cta, a.nsys - (int)blockIdx.x * u.per_cta);  // systems of this CTA
  const bool mine = g < nsys;
  double* base = reinterpret_cast<double*>(smem);
  double* sb = base + (size_t)(mine ? g : 0) * u.stride;
  double* PH = sb;            // p, then p_hat / s_hat
  double* RB = sb + n;        // r / s
  double* VB = sb + 2 * n;    // ISAI intermediate, then v / t (FP32 ISAI: input and intermediate, 2n floats)
  double* HB = sb + 3 * n;    // r_hat = b
  float* FI = reinterpret_cast<float*>(VB);
  float* FM = FI + n;
  const double* __restrict__ Am = a.A + (size_t)(mine ? sys : 0) * P.a_nnz;
  const FT* __restrict__ AL = reinterpret_cast<const FT*>(a.ail) + (size_t)(mine ? sys : 0) * P.ail_nnz;
  const FT* __restrict__ AU = reinterpret_cast<const FT*>(a.aiu) + (size_t)(mine ? sys : 0) * P.aiu_nnz;

  double x[R], r[R], p[R], v[R];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int i = t0 + k * ts;
    const double bi = mine && i < n ? __ldg(a.b + (size_t)sys * n + i) : 0.0;
    x[k] = 0.0;
    p[k] = 0.0;
    v[k] = 0.0;
    r[k] = bi;
    if (mine && i < n) HB[i] = bi;
  }
  __syncthreads();
  // ---- first warp: lane l < 8 owns system l's scalars; lanes 16 + l the second of two sums
  const bool ctl = tid < 32;
  const int lg = lane & 15;
  const bool lsys = lg < nsys;
  const double* cb = base + (size_t)(lsys ? lg : 0) * u.stride;
  const double *cPH = cb, *cRB = cb + n, *cVB = cb + 2 * n, *cHB = cb + 3 * n;
  (void)cPH;
  double rho = 0.0, rho_old = 1.0, alpha = 1.0, omega_old = 1.0, res = 0.0, thr = 0.0;
  float iter = 0.0f;
  int status = BILU_SYS_MAX_ITER;
  bool on = false;
  if (ctl) {
    const double d = lsys ? chain(cHB, cHB, n) : 0.0;
    const double nb = sqrt(d);
    res = nb;
    rho = d;  // (r, r_hat) of the first iteration: the same sum
    thr = a.tol_mode == BILU_TOL_ABS ? a.tol : a.tol * nb;
    on = lsys;
    if (nb == 0.0) {
      res = 0.0;
      status = BILU_SYS_ZERO_RHS;
      on = false;
    } else if (nb < thr) {
      status = BILU_SYS_INITIAL_OK;
      on = false;
    }
  }
  const float max_iter = (float)a.max_iter;
  // z = aiU (aiL in) into PH, the input in PH (FP64: p) / RB (FP64: s) / FI (FP32); ends with a barrier
  auto apply = [&](const double* in, bool act) {
    if (act) {
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int i = t0 + k * ts;
        if (i < n) {
          if constexpr (kFP32)
            FM[i] = row_seq(reinterpret_cast<const float*>(AL), P.ail_ci16, P.ail_rp, i, FI);
          else
            VB[i] = tree<SI, MI>(reinterpret_cast<const double*>(AL), P.ail_ci16, P.ail_rp, i, in);
        }
      }
    }
    __syncthreads();
    if (act) {
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int i = t0 + k * ts;
        if (i < n) {
          if constexpr (kFP32)
            PH[i] = (double)row_seq(reinterpret_cast<const float*>(AU), P.aiu_ci16, P.aiu_rp, i, FM);
          else
            PH[i] = tree<SI, MI>(reinterpret_cast<const double*>(AU), P.aiu_ci16, P.aiu_rp, i, VB);
        }
      }
    }
    __syncthreads();
  };
  // out = A PH, into VB too; ends with a barrier
  auto spmv = [&](double(&out)[R], bool act) {
    if (act) {
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int i = t0 + k * ts;
        if (i < n) {
          out[k] = tree<SA, MA>(Am, P.a_ci16, P.a_rp, i, PH);
          VB[i] = out[k];
        }
      }
    }
    __syncthreads();
  };
  for (;;) {
    // ---- loop head: breakdown, iteration limit, beta
    if (ctl) {
      if (on && !(iter < max_iter)) on = false;
      if (on && rho == 0.0) {
        status = BILU_SYS_BREAKDOWN_RHO;
        on = false;
      }
      const bool any = __any_sync(kFull, on);
      if (lane < kMaxSys) {
        s_a[lane] = on ? (rho / rho_old) * (alpha / omega_old) : 0.0;
        s_b[lane] = omega_old;
        s_on[lane] = on ? 1 : 0;
      }
      if (lane == 0) s_any = any ? 1 : 0;
    }
    __syncthreads();
    if (!s_any) break;
    bool act = mine && s_on[mine ? g : 0];
    if (act) {
      const double beta = s_a[g], om = s_b[g];
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int i = t0 + k * ts;
        if (i < n) {
          p[k] = fma(beta, fma(-om, v[k], p[k]), r[k]);
          if constexpr (kFP32)
            FI[i] = (float)p[k];
          else
            PH[i] = p[k];
        }
      }
    }
    __syncthreads();
    apply(PH, act);
    spmv(v, act);
    if (ctl) {
      const double d = on ? chain(cHB, cVB, n) : 1.0;
      alpha = on ? rho / d : alpha;
      if (lane < kMaxSys) s_a[lane] = alpha;
    }
    __syncthreads();
    if (act) {
      const double al = s_a[g];
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int i = t0 + k * ts;
        if (i < n) {
          x[k] = fma(al, PH[i], x[k]);
          r[k] = fma(-al, v[k], r[k]);
          RB[i] = r[k];
          if constexpr (kFP32) FI[i] = (float)r[k];
        }
      }
    }
    __syncthreads();
    if (ctl) {
      if (on) {
        res = sqrt(chain(cRB, cRB, n));
        iter = iter + 0.5f;
        if (res < thr) {
          status = BILU_SYS_CONVERGED;
          on = false;
        }
      }
      if (lane < kMaxSys) s_on[lane] = on ? 1 : 0;
    }
    __syncthreads();
    act = mine && s_on[mine ? g : 0];
    apply(RB, act);
    double t[R];
    spmv(t, act);
    if (ctl) {
      // lanes 0-15 (t, s), lanes 16-31 (t, t)
      const double d = on ? chain(cVB, lane < 16 ? cRB : cVB, n) : 1.0;
      const double tt = __shfl_down_sync(kFull, d, 16);
      const double om = __shfl_sync(kFull, d / tt, lg);  // both halves hold the system's omega
      if (on) {
        rho_old = rho;
        omega_old = om;
      }
      if (lane < kMaxSys) s_a[lane] = om;
    }
    __syncthreads();
    if (act) {
      const double om = s_a[g];
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int i = t0 + k * ts;
        if (i < n) {
          x[k] = fma(om, PH[i], x[k]);
          r[k] = fma(-om, t[k], r[k]);
          RB[i] = r[k];
        }
      }
    }
    __syncthreads();
    if (ctl) {
      // lanes 0-15 (r, r), lanes 16-31 the next iteration's (r, r_hat)
      const double d = on ? chain(cRB, lane < 16 ? cRB : cHB, n) : 0.0;
      const double rr = __shfl_sync(kFull, d, lg), rh = __shfl_sync(kFull, d, lg + 16);
      if (on) {
        res = sqrt(rr);
        rho = rh;
        iter = iter + 0.5f;
        if (res < thr) {
          status = BILU_SYS_CONVERGED;
          on = false;
        }
      }
    }
    // the loop head's barrier orders the next writes of RB and s_a after these reads
  }
  // ---- results
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int i = t0 + k * ts;
    if (mine && i < n) {
      a.x[(size_t)sys * n + i] = x[k];
      PH[i] = x[k];
    }
  }
  if (ctl && lane < nsys) {
    const int s = blockIdx.x * u.per_cta + lane;
    int st = status;
    if (st == BILU_SYS_MAX_ITER && !isfinite(res)) st = BILU_SYS_NONFINITE;
    const bool ok = st == BILU_SYS_CONVERGED || st == BILU_SYS_ZERO_RHS || st == BILU_SYS_INITIAL_OK;
    if (a.iters) a.iters[s] = iter;
    if (a.conv) a.conv[s] = ok ? 1 : -1;
    if (a.res) a.res[s] = res;
    if (a.status) a.status[s] = st;
  }
  // ---- true residual (KernelFillTrueResNorms, Bicgstab_common.hpp:294-342): b - A x, serial norm
  if (a.true_res) {
    __syncthreads();
    if (mine) {
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int i = t0 + k * ts;
        if (i < n) VB[i] = HB[i] - tree<SA, MA>(Am, P.a_ci16, P.a_rp, i, PH);
      }
    }
    __syncthreads();
    if (ctl && lane < nsys) a.true_res[blockIdx.x * u.per_cta + lane] = sqrt(chain(cVB, cVB, n));
  }
}

template <typename FT, int SA, int MA, int SI, int MI>
const void* by_rows(int R) {
  switch (R) {
    case 1: return (const void*)k_bicgstab_isai_ref<1, FT, SA, MA, SI, MI>;
    case 2: return (const void*)k_bicgstab_isai_ref<2, FT, SA, MA, SI, MI>;
    case 4: return (const void*)k_bicgstab_isai_ref<4, FT, SA, MA, SI, MI>;
    default: return (const void*)k_bicgstab_isai_ref<8, FT, SA, MA, SI, MI>;
  }
}

const void* pick(int R, int fp32, int maxa, int maxi) {
  if (fp32) return maxa <= 5 ? by_rows<float, 8, 5, 1, 1>(R) : maxa <= 7 ? by_rows<float, 8, 7, 1, 1>(R) : by_rows<float, 16, 16, 1, 1>(R);
  if (maxa <= 5 && maxi <= 6) return by_rows<double, 8, 5, 8, 6>(R);
  if (maxa <= 7 && maxi <= 10) return by_rows<double, 8, 7, 16, 10>(R);
  return by_rows<double, 16, 16, 16, 16>(R);
}

int stride_of(int n) { return 4 * n | 1; }

}  // namespace

bool isai_ref_fits(int n, int fp32, int maxa, int maxi) {
  return n <= 1024 && maxa <= 16 && (fp32 || maxi <= 16) && (long long)stride_of(n) * 8 <= 100 * 1024;
}

// Systems per CTA: the fewest that leave no more waves of CTAs (two per SM) than the most would, so that few
// systems spread over the SMs and a batch fills them evenly; rows per thread: the fewest that 256 threads allow.
cudaError_t launch_solve_isai_ref(const SolveArgs& a, int fp32, int maxa, int maxi, int nsm, cudaStream_t st) {
  if (a.nsys == 0) return cudaSuccess;
  const int n = a.pat.n, smax = std::min((int)(100 * 1024 / (8 * stride_of(n))), kMaxSys);
  const int gmax = std::max(1, std::min(smax, 8 / ((n + 255) / 256)));
  const long long slots = 2LL * nsm;
  const long long waves = (a.nsys + slots * gmax - 1) / (slots * gmax);
  IsaiRefArgs u;
  u.s = a;
  u.per_cta = (int)std::max(1LL, std::min((long long)gmax, (a.nsys + slots * waves - 1) / (slots * waves)));
  int R = 1;
  while ((n + 32 * R - 1) / (32 * R) * u.per_cta > kThreads / 32) R *= 2;
  u.tsys = (n + 32 * R - 1) / (32 * R) * 32;
  u.stride = stride_of(n);
  const void* k = pick(R, fp32, maxa, maxi);
  const int smem = u.stride * 8 * u.per_cta;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  void* args[] = {&u};
  return cudaLaunchKernel(k, dim3((a.nsys + u.per_cta - 1) / u.per_cta), dim3(u.tsys * u.per_cta), args, (size_t)smem, st);
}

}  // namespace bilu
