// The plain form's solver: one warp per world in index order, the Hessian refactored every iteration.
#include "mjb_solver_queue.cuh"

namespace mjb {

__global__ void __launch_bounds__(128, MJB_MINB) k_solve_plain(const __grid_constant__ MjbModel m, const __grid_constant__ MjbData d, int smem_per_warp) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= d.nworld) return;
  float* sm = smem_per_warp ? smem + size_t(threadIdx.x >> 5) * smem_per_warp : nullptr;
  solve(m, d, w, lane, sm, d.efc_h + W(w, m.nv * m.nv));
}

int launch_solver_plain(const MjbModel* m, const MjbData* d, cudaStream_t s) {
  const int spw = m->nv <= 32 ? int(solver_smem_floats(m->nv)) : generic_nz_floats(m->nv);
  const size_t bytes = size_t(spw) * kDefaultWarps * sizeof(float);
  if (bytes > kMaxSmemPerCta) return MJB_ERR_SCRATCH;
  static size_t configured[kSmemDevices];
  allow_smem(k_solve_plain, bytes, configured);
  k_solve_plain<<<grid_for(d->nworld, kDefaultWarps), 32 * kDefaultWarps, bytes, s>>>(*m, *d, spw);
  return finish();
}

}  // namespace mjb
