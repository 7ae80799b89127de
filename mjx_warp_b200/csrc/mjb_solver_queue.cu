// The chosen form's persistent solver, FP32 FMAs, 5 CTAs per SM.
#include "mjb_solver_queue.cuh"

namespace mjb {

void launch_solver_warp(const MjbModel* m, const MjbData* d, int warps, int spw, cudaStream_t s) {
  launch_warp<false, false, 5>(m, d, warps, spw, s);
}

}  // namespace mjb
