// The chosen form's persistent solver at 4 CTAs per SM, with FMAs or the Hessian on the tensor pipe.
#include "mjb_solver_queue.cuh"

namespace mjb {

void launch_solver_warp_alt(const MjbModel* m, const MjbData* d, bool tc, int warps, int spw, cudaStream_t s) {
  if (tc) launch_warp<false, true, MJB_MINB>(m, d, warps, spw, s);
  else if (scheduled(d)) launch_solver_queue<false, false, 4>(m, d, warps, spw, s);
  else launch_solver_warp(m, d, warps, spw, s);  // one kernel for both, mjb_solver_queue.cu's
}

}  // namespace mjb
