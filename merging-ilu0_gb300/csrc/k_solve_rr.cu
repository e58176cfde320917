// Register-resident batched BiCGSTAB: the main kernel (one CTA per system of
// a batch sharing one pattern) and the launch code; the device code is in
// k_solve_rr.cuh, the occupancy variants in k_solve_rr_occ.cu and the
// uneven-batch kernel in k_solve_rr_uneven.cu.
#include "k_solve_rr.cuh"

namespace bilu {
namespace {

// one CTA per system of a batch sharing one pattern
// ORD = kRef, kRefLean: the reference's operation order.  Warp w's lane l owns
// rows l + 32 (w R + k), a block of the reference's lane-strided inner-product
// terms; the inner products chain through the warps in order (ref_chain_sum),
// so every scalar is the reference's bit for bit.
template <int R, int PV, typename FT, int ORD>
__global__ void BILU_RR_BOUNDS k_bicgstab_rr(const SolveArgs a, const RRLayout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int sys = blockIdx.x;
  if (sys >= a.nsys) return;
  const DevPattern& P = a.pat;
  rr_solve<R, PV, FT, true, ORD>(a, P, L, smem, sys, a.A + (size_t)sys * P.a_nnz, a.b + (size_t)sys * P.n,
                                 a.x + (size_t)sys * P.n);
}

template <int PV, typename FT, int ORD>
const void* rr_kernel_pv(int slots) {
  switch (slots) {
    case 1: return (const void*)k_bicgstab_rr<1, PV, FT, ORD>;
    case 2: return (const void*)k_bicgstab_rr<2, PV, FT, ORD>;
    case 3: return (const void*)k_bicgstab_rr<3, PV, FT, ORD>;
    case 4: return (const void*)k_bicgstab_rr<4, PV, FT, ORD>;
  }
  if constexpr (PV == 3 || PV == 0 || ORD != kFast)  // else split (rr_split)
    return slots == 6 ? (const void*)k_bicgstab_rr<6, PV, FT, ORD> : (const void*)k_bicgstab_rr<8, PV, FT, ORD>;
  return nullptr;
}

}  // namespace

int rr_rows_per_thread(int n, int nt) {
  for (int R : {1, 2, 4, 8})
    if ((long long)R * nt >= n) return R;
  return 0;
}

int rr_slots(int n, int nt) {
  for (int R : {1, 2, 3, 4, 6, 8})
    if ((long long)R * nt >= n) return R;
  return 0;
}

int rr_max_threads(int R, bool wide) {
  if (wide) return R == 8 ? 256 : 0;
  return R <= 1 ? 1024 : (R == 2 ? 512 : (R == 4 ? 256 : 128));
}

// Threads per order thread (k_bicgstab_rr_split): FAST order without ILU
// factors at 5 to 8 rows per thread.  Four while every system then is resident
// at once (64 registers: 1024 threads per SM), where a system's own latency is
// all that counts: 16 systems of 3D 10x10x10, FP32 ISAI, 0.375 ms on one, 0.336
// on two, 0.246 on four; 300 systems 0.495 / 0.449 / 0.352; 450, which four
// leave waiting, 0.543 / 0.474 / 0.580.  Past that two, but for 7 or 8 rows on
// one warp (8192 2D 16x16 systems 1.64 ms on two, 1.47 on four; at 96 and 128
// threads four are 5 to 15 % slower).
//
// Without a preconditioner (pv = 0) the inner products, which a split lengthens,
// are most of an iteration: at 128 threads four only while each system has an SM
// to itself, and two instead of one only where the 1024 / (2 nt) CTAs that then
// share an SM, instead of 384 / nt, save a wave that outweighs a wave's 1.1 to
// 1.3 times longer time; past four waves the two forms are within 5 % of each
// other either way.  Microseconds on one / two / four, 31x31: 152 systems 168 /
// 166 / 154, 304 197 / 209 / 199, 456 243 / 263 / 375, 608 451 / 326 / 389, 800 467
// / 530 / 567, 2048 1127 / 1156 / 1304; 760 tridiagonal rows, 96 threads: 304 193 /
// 206 / 187, 1000 488 / 550 / 656, 1500 714 / 651 / 847.  On one warp one while
// it is a single wave: 16x16, 1500 systems 241 / 244 / 300, 2048 418 / 335 / 364.
int rr_split(int pv, int ref, int n, int nt, int nsys, int nsm) {
  const int slots = rr_slots(n, nt);
  if (pv == 3 || ref || slots < 6 || nt > 128) return 1;
  if (nsys <= (long long)nsm * (pv == 0 && nt == 128 ? 1 : 1024 / (4 * nt))) return 4;
  auto waves = [&](long long per) { return (nsys + per * nsm - 1) / (per * nsm); };
  const long long one = waves(384 / nt), two = waves(1024 / (2 * nt));
  if (slots == 8 && nt == 32) return pv == 0 && one == 1 ? 1 : 4;
  if (pv != 0) return 2;
  return one <= 4 && 10 * one >= 13 * two ? 2 : 1;
}

const void* rr_kernel(int pv, int fp32, int n, int nt, int ref, int occ, int mc, int split) {
  const int slots = rr_slots(n, nt);
  if (nt > 128 && slots > 4) return occ ? nullptr : rr_wide_kernel(pv, fp32, ref, nt, mc);
  if (split > 1) return rr_split_kernel(pv, fp32, split, slots);
  if (occ && slots <= 4) return ref ? nullptr : rr_occ_kernel(pv, fp32, slots);  // FAST order, 2 to 4 rows
  if (pv == 3 && mc) return rr_lu_kernel(fp32, slots, ref, mc);
  if (ref) {  // reference order: no preconditioner or ILU factors
    if (pv == 0) return rr_kernel_pv<0, double, kRef>(slots);
    if (pv != 3) return nullptr;
    if (ref == kRefLean)  // 5 to 8 rows per thread (rr_configure)
      return slots == 6 ? (const void*)k_bicgstab_rr<6, 3, double, kRefLean>
                        : (const void*)k_bicgstab_rr<8, 3, double, kRefLean>;
    return fp32 ? rr_kernel_pv<3, float, kRef>(slots) : rr_kernel_pv<3, double, kRef>(slots);
  }
  if (pv == 0) return rr_kernel_pv<0, double, kFast>(slots);
  if (pv == 1) return fp32 ? rr_kernel_pv<1, float, kFast>(slots) : rr_kernel_pv<1, double, kFast>(slots);
  if (pv == 3) return fp32 ? rr_kernel_pv<3, float, kFast>(slots) : rr_kernel_pv<3, double, kFast>(slots);
  return fp32 ? rr_kernel_pv<2, float, kFast>(slots) : rr_kernel_pv<2, double, kFast>(slots);
}

const char* rr_kernel_name(int pv, int n, int nt, int ref, int occ, int mc, int nsys, int nsm) {
  const int slots = rr_slots(n, nt);
  if (nt > 128 && slots > 4) return "k_bicgstab_rr_wide";
  if (rr_split(pv, ref, n, nt, nsys, nsm) > 1) return "k_bicgstab_rr_split";
  if (occ && slots <= 4) return "k_bicgstab_rr_occ";
  return pv == 3 && mc ? "k_bicgstab_rr_lu" : "k_bicgstab_rr";
}

cudaError_t launch_solve_rr(const SolveArgs& a, const RRLayout& L, int nt, int pv, int fp32, int ref, int occ,
                            int nsm, cudaStream_t st) {
  if (a.nsys == 0) return cudaSuccess;
  const int R = rr_rows_per_thread(a.pat.n, nt);
  if (R == 0 || nt % 32 || nt > rr_max_threads(R, a.pat.n > 1024)) return cudaErrorInvalidConfiguration;
  const int split = rr_split(pv, ref, a.pat.n, nt, a.nsys, nsm);
  const void* k = rr_kernel(pv, fp32, a.pat.n, nt, ref, occ, a.pat.tc_mc, split);
  if (!k) return cudaErrorInvalidConfiguration;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, L.total);
  if (e != cudaSuccess) return e;
  void* args[] = {const_cast<SolveArgs*>(&a), const_cast<RRLayout*>(&L)};
  return cudaLaunchKernel(k, dim3(a.nsys), dim3(nt * split), args, (size_t)L.total, st);
}

}  // namespace bilu
