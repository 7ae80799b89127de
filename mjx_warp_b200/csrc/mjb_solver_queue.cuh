// The persistent one-warp-per-world solver kernels and their launch, instantiated by the units that
// mjb_launch.cuh names.
#pragma once

#include "mjb_launch.cuh"
#include "mjb_solver.cuh"

// minimum resident CTAs per SM requested for the solver kernels (caps registers per thread at
// 65536 / (128 * MJB_MINB)); with the staged / unstaged solver paths compiled apart, 4 (128
// registers) measured 2 % faster than 5 (96 registers, spilling) on the humanoid at 8192 worlds
#ifndef MJB_MINB
#define MJB_MINB 4
#endif
// The chosen form's FP32 persistent solver (k_solve_queue<false, false, *>) is compiled for 4 and for
// 5 (MjbTune.solver_ctas_per_sm): on the humanoid at 8192 worlds 5 CTAs per SM (96 registers, with
// spills) measured 0.241 against 0.256 ms early in a run and 0.381 against 0.352 ms once the worlds
// lie on the floor; the plain form's solver and the precision solver were slower at 5.

namespace mjb {

// chosen form: the constraint solver with the Hessian factor kept across iterations; TC: the
// Newton Hessian of up to 32 staged rows assembled on the tensor pipe in split TF32 (hessian_tc;
// always in the precision form, an autotuner choice in the chosen form)
template <bool PREC, bool TC>
__global__ void __launch_bounds__(128, MJB_MINB) k_solve(const __grid_constant__ MjbModel m, const __grid_constant__ MjbData d, int smem_per_warp) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= d.nworld) return;
  float* sm = smem_per_warp ? smem + size_t(threadIdx.x >> 5) * smem_per_warp : nullptr;
  solve<PREC, TC>(m, d, w, lane, sm, d.efc_h + W(w, m.nv * m.nv), true);
}

// persistent over k_order_worlds' order: each warp takes the next world from the queue
template <bool PREC, bool TC, int MINB>
__global__ void __launch_bounds__(128, MINB) k_solve_queue(const __grid_constant__ MjbModel m, const __grid_constant__ MjbData d, int smem_per_warp) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31;
  float* sm = smem_per_warp ? smem + size_t(threadIdx.x >> 5) * smem_per_warp : nullptr;
  for (;;) {
    int idx = 0;
    if (lane == 0) idx = atomicAdd(d.work_queue, 1);
    idx = __shfl_sync(WARP_FULL, idx, 0);
    if (idx >= d.nworld) break;
    const int w = d.world_order[idx];
    solve<PREC, TC>(m, d, w, lane, sm, d.efc_h + W(w, m.nv * m.nv), true);
  }
}

template <bool PREC, bool TC, int MINB>
inline void launch_solver_queue(const MjbModel* m, const MjbData* d, int qw, int spw, cudaStream_t s) {
  const size_t qbytes = size_t(spw) * qw * sizeof(float);
  static size_t conf_queue[kSmemDevices];
  allow_smem(k_solve_queue<PREC, TC, MINB>, size_t(spw) * kDefaultWarps * sizeof(float), conf_queue);
  const int ctas = resident_ctas(k_solve_queue<PREC, TC, MINB>, 32 * qw, qbytes);  // ordered in phase 0
  k_solve_queue<PREC, TC, MINB><<<std::min(ctas, grid_for(d->nworld, qw)), 32 * qw, qbytes, s>>>(*m, *d, spw);
}

// the persistent kernel when the Data has the schedule arrays, else one warp per world
template <bool PREC, bool TC, int MINB>
inline void launch_warp(const MjbModel* m, const MjbData* d, int warps, int spw, cudaStream_t s) {
  if (d->world_order && d->work_queue && d->world_nefc) {
    launch_solver_queue<PREC, TC, MINB>(m, d, warps, spw, s);
  } else {
    const size_t bytes = size_t(spw) * kDefaultWarps * sizeof(float);
    static size_t conf_solve[kSmemDevices];
    allow_smem(k_solve<PREC, TC>, bytes, conf_solve);
    k_solve<PREC, TC><<<grid_for(d->nworld, kDefaultWarps), 32 * kDefaultWarps, bytes, s>>>(*m, *d, spw);
  }
}

}  // namespace mjb
