// Register-resident solver in FAST order at 5 to 8 rows per order thread (ISAI,
// general ISAI or no preconditioner): SPLIT threads share an order thread's
// rows (split_chain_sum, k_solve_rr.cuh), so the order and every bit stay those
// of nt threads while the registers per thread halve and twice or four times
// as many warps cover the FP64, L1 and barrier latencies that bound the solve
// (12 warps per SM at 168 registers issued 57 % of the FP64 pipe).  RP = rows
// per thread: three for 5 or 6 rows, so that no row slot past the system's is
// issued predicated off, each FP64 instruction of which takes its slot.
// Measured, solver alone, one thread per order thread -> this: ILU(0) + FP32
// ISAI of 16384 23x25 systems 17.8 -> 12.8 ms; of 8192 3D 7x7x7 systems 2.95 ->
// 2.12 ms; of 4096 3D 10x10x10 systems 4.23 -> 3.52 ms; of 16 of them 0.375 ->
// 0.246 ms.  Bounds for five CTAs per SM instead of four spill: 23x25 13.8 ms.
#include "k_solve_rr.cuh"

namespace bilu {
namespace {

template <int SPLIT, int RP, int PV, typename FT>
__global__ void __launch_bounds__(128 * SPLIT, SPLIT == 2 ? 4 : 2) k_bicgstab_rr_split(const SolveArgs a,
                                                                                      const RRLayout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int sys = blockIdx.x;
  if (sys >= a.nsys) return;
  const DevPattern& P = a.pat;
  rr_solve<RP, PV, FT, true, kFast, false, 0, SPLIT>(a, P, L, smem, sys, a.A + (size_t)sys * P.a_nnz,
                                                     a.b + (size_t)sys * P.n, a.x + (size_t)sys * P.n);
}

template <int PV, typename FT>
const void* split_pv(int split, int slots) {
  if (split == 4) return (const void*)k_bicgstab_rr_split<4, 2, PV, FT>;
  return slots == 6 ? (const void*)k_bicgstab_rr_split<2, 3, PV, FT> : (const void*)k_bicgstab_rr_split<2, 4, PV, FT>;
}

}  // namespace

const void* rr_split_kernel(int pv, int fp32, int split, int slots) {
  if (pv == 0) return split_pv<0, double>(split, slots);
  if (pv == 1) return fp32 ? split_pv<1, float>(split, slots) : split_pv<1, double>(split, slots);
  if (pv == 2) return fp32 ? split_pv<2, float>(split, slots) : split_pv<2, double>(split, slots);
  return nullptr;
}

}  // namespace bilu
