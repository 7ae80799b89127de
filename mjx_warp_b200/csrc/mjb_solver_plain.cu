// The plain form's solver: one warp per world in index order, the Hessian refactored every iteration.
#include "mjb_solver_queue.cuh"

namespace mjb {

// SMALL: small_model's solver, else the generic one; in one kernel they hold each other's registers
template <bool SMALL>
__global__ void __launch_bounds__(128, MJB_MINB) k_solve_plain(const __grid_constant__ MjbModel m, const __grid_constant__ MjbData d, int smem_per_warp) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= d.nworld) return;
  float* sm = smem + size_t(threadIdx.x >> 5) * smem_per_warp;
  if constexpr (SMALL) solve_small(m, d, w, lane, sm, false);
  else solve_generic(m, d, w, lane, d.efc_h + W(w, m.nv * m.nv), sm, false);
}

template <bool SMALL>
static int launch_plain(const MjbModel* m, const MjbData* d, int spw, cudaStream_t s) {
  const size_t bytes = size_t(spw) * kDefaultWarps * sizeof(float);
  if (bytes > kMaxSmemPerCta) return MJB_ERR_SCRATCH;
  static size_t configured[kSmemDevices];
  allow_smem(k_solve_plain<SMALL>, bytes, configured);
  k_solve_plain<SMALL><<<grid_for(d->nworld, kDefaultWarps), 32 * kDefaultWarps, bytes, s>>>(*m, *d, spw);
  return finish();
}

int launch_solver_plain(const MjbModel* m, const MjbData* d, cudaStream_t s) {
  return small_model(*m) ? launch_plain<true>(m, d, int(solver_smem_floats(m->nv)), s)
                         : launch_plain<false>(m, d, generic_nz_floats(m->nv), s);
}

}  // namespace mjb
