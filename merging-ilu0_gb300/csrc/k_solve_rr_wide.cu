// Register-resident solver for systems of 1025 to 2048 rows (k_solve_rr.cuh),
// in a translation unit of its own so that it compiles in parallel with the
// rest: 8 rows per thread, ILU factors or no preconditioner, in the reference's
// order or the FAST order that these systems have always had (kFastChain), so
// the bits are those of the shared-memory solver (k_solve.cu).
//
// What bounds these systems is the latency of their level-scheduled solves (71
// levels per triangle at 36x36).  The shared-memory solver keeps seven vectors,
// A and the factors in shared memory, one CTA of 1024 threads per SM, and
// every level chases its metadata through L2 and ends in a barrier; here the
// vectors are in registers, the solves run from the prefetched programs on as
// many warps as a level has rows, and several systems share an SM: ParILU(5)
// solve of 512 36x36 systems, reference order, 13.6 -> 4.2 ms, and 3.5 ms with
// the compact programs.
#include "k_solve_rr.cuh"

namespace bilu {
namespace {

// Two CTAs per SM without spills to speak of (168 registers at 192 threads, n
// <= 1536; 128 at 256).  Three CTAs at 192 threads spill 500 bytes per thread:
// ParILU(5) of 512 36x36 systems 5.48 ms instead of 4.16.
template <int NT, int PV, typename FT, int ORD, int MC>
__global__ void __launch_bounds__(NT, 2) k_bicgstab_rr_wide(const SolveArgs a, const RRLayout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int sys = blockIdx.x;
  if (sys >= a.nsys) return;
  const DevPattern& P = a.pat;
  rr_solve<8, PV, FT, true, ORD, true, MC>(a, P, L, smem, sys, a.A + (size_t)sys * P.a_nnz, a.b + (size_t)sys * P.n,
                                       a.x + (size_t)sys * P.n);
}

template <int PV, typename FT, int MC = 0>
const void* wide_pv(int ref, int nt) {
  if (nt <= 192)
    return ref ? (const void*)k_bicgstab_rr_wide<192, PV, FT, kRefLean, MC>
               : (const void*)k_bicgstab_rr_wide<192, PV, FT, kFastChain, MC>;
  return ref ? (const void*)k_bicgstab_rr_wide<256, PV, FT, kRefLean, MC>
             : (const void*)k_bicgstab_rr_wide<256, PV, FT, kFastChain, MC>;
}

template <int MC>
const void* wide_lu(int fp32, int ref, int nt) {
  return fp32 ? wide_pv<3, float, MC>(ref, nt) : wide_pv<3, double, MC>(ref, nt);
}

}  // namespace

const void* rr_wide_kernel(int pv, int fp32, int ref, int nt, int mc) {
  if (pv == 0) return wide_pv<0, double>(ref, nt);
  if (pv == 3) return mc == 2 ? wide_lu<2>(fp32, ref, nt) : mc == 3 ? wide_lu<3>(fp32, ref, nt) : wide_lu<0>(fp32, ref, nt);
  return nullptr;
}

}  // namespace bilu
