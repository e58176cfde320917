// Register-resident solver with ILU factors whose triangles have at most two or
// three entries per row (2D 5-point and 3D 7-point stencils): the solves run
// from the compact programs (tri_solve_compact, k_solve_rr.cuh).  Kernels of
// their own rather than a branch in k_bicgstab_rr, because a second copy of the
// solves in one kernel slowed both (k_solve_rr.cuh, team_sync).  Bound by FP64
// issue and the levels' latency.  Against the general programs: merged ILU(0)
// of 4096 3D 10x10x10 systems, FAST order, 6.26 -> 5.43 ms; of 4096 2D 16x16
// systems in the reference's order 3.08 -> 2.92 ms, of 8 2D 8x8 systems 276 ->
// 224 us.  With the merged form's ILU(0) from its compact program too
// (ilu_compact_rows) 5.45 -> 5.14 ms, 2.92 -> 2.78 ms, 224 -> 217 us.
#include "k_solve_rr.cuh"

namespace bilu {
namespace {

template <int R, typename FT, int ORD, int MC>
__global__ void BILU_RR_BOUNDS k_bicgstab_rr_lu(const SolveArgs a, const RRLayout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int sys = blockIdx.x;
  if (sys >= a.nsys) return;
  const DevPattern& P = a.pat;
  rr_solve<R, 3, FT, true, ORD, false, MC>(a, P, L, smem, sys, a.A + (size_t)sys * P.a_nnz, a.b + (size_t)sys * P.n,
                                           a.x + (size_t)sys * P.n);
}

template <typename FT, int ORD, int MC>
const void* lu_r(int slots) {
  switch (slots) {
    case 1: return (const void*)k_bicgstab_rr_lu<1, FT, ORD, MC>;
    case 2: return (const void*)k_bicgstab_rr_lu<2, FT, ORD, MC>;
    case 3: return (const void*)k_bicgstab_rr_lu<3, FT, ORD, MC>;
    case 4: return (const void*)k_bicgstab_rr_lu<4, FT, ORD, MC>;
    case 6: return (const void*)k_bicgstab_rr_lu<6, FT, ORD, MC>;
    default: return (const void*)k_bicgstab_rr_lu<8, FT, ORD, MC>;
  }
}

template <int MC>
const void* lu_mc(int fp32, int slots, int ref) {
  if (ref == kRefLean)  // 5 to 8 rows per thread (rr_configure)
    return slots == 6 ? (const void*)k_bicgstab_rr_lu<6, double, kRefLean, MC>
                      : (const void*)k_bicgstab_rr_lu<8, double, kRefLean, MC>;
  if (ref) return fp32 ? lu_r<float, kRef, MC>(slots) : lu_r<double, kRef, MC>(slots);
  return fp32 ? lu_r<float, kFast, MC>(slots) : lu_r<double, kFast, MC>(slots);
}

}  // namespace

const void* rr_lu_kernel(int fp32, int slots, int ref, int mc) {
  return mc == 2 ? lu_mc<2>(fp32, slots, ref) : lu_mc<3>(fp32, slots, ref);
}

}  // namespace bilu
