// The precision form's persistent solver for nv <= 32.
#include "mjb_solver_queue.cuh"

namespace mjb {

void launch_solver_warp_prec(const MjbModel* m, const MjbData* d, int warps, int spw, cudaStream_t s) {
  launch_warp<true, true, MJB_MINB>(m, d, warps, spw, s);
}

}  // namespace mjb
