// The CTA-per-world solver's kernels and their launch (mjb_solver_cta.cuh), instantiated for FP32 by
// mjb_solver_cta.cu and for the precision form by mjb_solver_cta_prec.cu.
#pragma once

#include "mjb_launch.cuh"
#include "mjb_solver_cta.cuh"

namespace mjb {

// chosen form, models with nv > 32: one CTA of NW warps per world (mjb_solver_cta.cuh),
// persistent over the work queue in k_order_worlds' order when the Data has the schedule arrays,
// else one CTA per world in index order
template <int NW, bool PREC, bool TREES>
__global__ void __launch_bounds__(NW * 32, NW >= 16 ? 1 : (NW >= 8 ? 2 : (NW >= 4 ? 4 : (NW >= 2 ? 8 : 9))))
    k_solve_cta(const __grid_constant__ MjbModel m, const __grid_constant__ MjbData d, int tc) {
  extern __shared__ __align__(16) float smem[];
  __shared__ int s_idx;
  if (!d.work_queue) {
    if (int(blockIdx.x) < d.nworld) solve_cta<NW, PREC, TREES>(m, d, blockIdx.x, smem, tc != 0);
    return;
  }
  for (;;) {
    if (threadIdx.x == 0) s_idx = atomicAdd(d.work_queue, 1);
    __syncthreads();
    const int idx = s_idx;
    __syncthreads();
    if (idx >= d.nworld) break;
    solve_cta<NW, PREC, TREES>(m, d, d.world_order[idx], smem, tc != 0);
  }
}

template <int NW, bool PREC, bool TREES>
inline void launch_cta_form(const MjbModel* m, const MjbData* d, int tc, cudaStream_t s) {
  const size_t bytes = size_t(cta_solver_smem_floats(m->nv, NW, PREC, TREES)) * sizeof(float);
  static size_t conf[kSmemDevices];
  allow_smem(k_solve_cta<NW, PREC, TREES>, bytes, conf);
  if (scheduled(d)) {
    const int ctas = resident_ctas(k_solve_cta<NW, PREC, TREES>, 32 * NW, bytes);  // ordered in phase 0
    k_solve_cta<NW, PREC, TREES><<<std::min(ctas, d->nworld), 32 * NW, bytes, s>>>(*m, *d, tc);
  } else {
    MjbData dd = *d;
    dd.work_queue = nullptr;
    k_solve_cta<NW, PREC, TREES><<<d->nworld, 32 * NW, bytes, s>>>(*m, dd, tc);
  }
}

template <int NW, bool PREC>
inline void launch_cta(const MjbModel* m, const MjbData* d, int tc, cudaStream_t s) {
  if constexpr (!PREC) {
    if (NW == 1 || sparse_launch<NW>(*m, tc != 0)) return launch_cta_form<NW, PREC, true>(m, d, tc, s);
  }
  if constexpr (NW > 1) launch_cta_form<NW, PREC, false>(m, d, tc, s);
}

}  // namespace mjb
