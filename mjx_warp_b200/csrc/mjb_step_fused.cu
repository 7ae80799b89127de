// The single form: the whole step of a world in one warp of one kernel.
#include "mjb_solver_queue.cuh"
#include "mjb_state.cuh"

namespace mjb {

// whole forward (+ integration) of one world per warp; each warp's slice of dynamic shared memory
// holds the solver's workspace, whose leading factor tile also serves the mass-matrix
// factorisations (factor_m, then the integrator).  SMALL: small_model's solver, else the generic one
template <bool SMALL>
__global__ void __launch_bounds__(128, MJB_MINB) k_step_fused(const __grid_constant__ MjbModel m, const __grid_constant__ MjbData d, int integrate,
                                                    int smem_per_warp) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int w = blockIdx.x * (blockDim.x >> 5) + wib;
  if (w >= d.nworld) return;
  const int nv = m.nv;
  float* sm = smem_per_warp ? smem + size_t(wib) * smem_per_warp : nullptr;
  [[maybe_unused]] float* hs = d.efc_h + W(w, nv * nv);
  kinematics(m, d, w, lane);
  com_pos(m, d, w, lane);
  crb(m, d, w, lane);
  factor_m(m, d, w, lane, sm);
  collision(m, d, w, lane, sm);
  make_constraint(m, d, w, lane);
  transmission(m, d, w, lane);
  fwd_velocity(m, d, w, lane);
  fwd_actuation(m, d, w, lane);
  fwd_acceleration(m, d, w, lane, sm, true);  // the tile still holds factor_m's factor
  if (d.njmax == 0) copy_qacc_smooth(m, d, w, lane);
  else if constexpr (SMALL) solve_small(m, d, w, lane, sm, true);
  else solve_generic(m, d, w, lane, hs, sm, true);
  if (integrate) {
    if (m.integrator == 0) euler(m, d, w, lane, sm);
    else implicit(m, d, w, lane, sm);
    check_finite(m, d, w, lane);
  }
}

void launch_step_fused(const MjbModel* m, const MjbData* d, int integrate, int warps, int spw, size_t smem, cudaStream_t s) {
  static size_t configured[2][kSmemDevices];
  const bool small = small_model(*m);
  const auto k = small ? k_step_fused<true> : k_step_fused<false>;
  allow_smem(k, smem, configured[small]);
  k<<<grid_for(d->nworld, warps), 32 * warps, smem, s>>>(*m, *d, integrate, spw);
}

}  // namespace mjb
