// The persistent one-warp-per-world solver kernels for nv <= 32 with a dense mass matrix, and their launch,
// instantiated by the units that mjb_launch.cuh names.
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
// 5 (MjbTune.solver_ctas_per_sm).  The default is 4: with the rarer paths in a kernel of their own 128
// registers hold the path with few spills, and on the humanoid at 8192 worlds the solver takes 0.230
// against 0.243 ms over the first 20 steps and 0.376 against 0.390 after 200 (one kernel with every path:
// 0.256 against 0.241 at first, so 5 was the default then); the step with up to 44 rows 484 against 497
// us, 1000 worlds 275 against 300, 32768 2162 against 2262.  The plain form's solver and the precision
// solver were slower at 5.

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
  solve_small<PREC, TC>(m, d, w, lane, sm, true);
}

// persistent over k_order_worlds' order: each warp takes the next world from the queue.  ALL: every
// solver and search; else only Newton with the iterative search (queue_newton), without the registers
// and the instructions of the rest (560 bytes of spill loads against 864).  With the generic solver in a
// unit of its own, 8192 humanoid worlds of a few rows each: solver 0.250 -> 0.243 ms, precision form's step
// 0.89 -> 0.85; with up to 44 rows, step 507 -> 497 us, 32768 worlds 2290 -> 2245.
template <bool PREC, bool TC, int MINB, bool ALL>
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
    solve_small<PREC, TC, ALL>(m, d, w, lane, sm, true);
  }
}

inline bool queue_newton(const MjbModel* m) { return m->solver != 1 && !m->ls_parallel; }

template <bool PREC, bool TC, int MINB, bool ALL>
inline void launch_queue_form(const MjbModel* m, const MjbData* d, int qw, int spw, cudaStream_t s) {
  const size_t qbytes = size_t(spw) * qw * sizeof(float);
  static size_t conf_queue[kSmemDevices];
  allow_smem(k_solve_queue<PREC, TC, MINB, ALL>, size_t(spw) * kDefaultWarps * sizeof(float), conf_queue);
  const int ctas = resident_ctas(k_solve_queue<PREC, TC, MINB, ALL>, 32 * qw, qbytes);  // ordered in phase 0
  k_solve_queue<PREC, TC, MINB, ALL><<<std::min(ctas, grid_for(d->nworld, qw)), 32 * qw, qbytes, s>>>(*m, *d, spw);
}

template <bool PREC, bool TC, int MINB>
inline void launch_solver_queue(const MjbModel* m, const MjbData* d, int qw, int spw, cudaStream_t s) {
  if (queue_newton(m)) launch_queue_form<PREC, TC, MINB, false>(m, d, qw, spw, s);
  else launch_queue_form<PREC, TC, MINB, true>(m, d, qw, spw, s);
}

// the persistent kernel when the Data has the schedule arrays, else one warp per world
template <bool PREC, bool TC, int MINB>
inline void launch_warp(const MjbModel* m, const MjbData* d, int warps, int spw, cudaStream_t s) {
  if (scheduled(d)) {
    launch_solver_queue<PREC, TC, MINB>(m, d, warps, spw, s);
  } else {
    const size_t bytes = size_t(spw) * kDefaultWarps * sizeof(float);
    static size_t conf_solve[kSmemDevices];
    allow_smem(k_solve<PREC, TC>, bytes, conf_solve);
    k_solve<PREC, TC><<<grid_for(d->nworld, kDefaultWarps), 32 * kDefaultWarps, bytes, s>>>(*m, *d, spw);
  }
}

}  // namespace mjb
