// The chosen form's persistent solver at 4 CTAs per SM, with FMAs or the Hessian on the tensor pipe.
#include "mjb_solver_queue.cuh"

namespace mjb {

void launch_solver_warp_alt(const MjbModel* m, const MjbData* d, bool tc, int warps, int spw, cudaStream_t s) {
  if (tc) launch_warp<false, true, MJB_MINB>(m, d, warps, spw, s);
  else launch_warp<false, false, 4>(m, d, warps, spw, s);
}

}  // namespace mjb
