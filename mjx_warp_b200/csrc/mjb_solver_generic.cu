// The generic solver's kernels, one warp per world: models of one tree past 32 dofs, larger ones where the
// tuning asks for one warp, the sparse mass matrix up to 32 dofs.  A unit of its own: in one kernel with
// the small models' solver the two held each other's registers.  Four blocks of four warps per SM (128
// registers): forward of 4096 worlds of a 40-dof chain 7.4 ms against 8.1 with five, of 2048 worlds of a
// 100-dof chain 22.7 against 22.5, of 2048 worlds of 20 boxes 10.5 against 10.6.
#include "mjb_launch.cuh"
#include "mjb_solver.cuh"

namespace mjb {

// persistent over k_order_worlds' order: each warp takes the next world from the queue
__global__ void __launch_bounds__(128, 4) k_solve_generic_queue(const __grid_constant__ MjbModel m, const __grid_constant__ MjbData d, int smem_per_warp) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31;
  float* sm = smem + size_t(threadIdx.x >> 5) * smem_per_warp;
  for (;;) {
    int idx = 0;
    if (lane == 0) idx = atomicAdd(d.work_queue, 1);
    idx = __shfl_sync(WARP_FULL, idx, 0);
    if (idx >= d.nworld) break;
    const int w = d.world_order[idx];
    solve_generic(m, d, w, lane, d.efc_h + W(w, m.nv * m.nv), sm, true);
  }
}

// The worlds of more than min_rows rows, without the queue.  With the schedule arrays they come first in
// the order (its buckets tell up to 254 rows apart, min_rows < 254), so every warp stops at its first
// smaller one.  Beside k_solve_cta<1>, which leaves them out: there a world takes 24 KB of shared memory,
// so nine warps run on an SM, here sixteen.  2048 worlds of 20 boxes lying on a plane (320 rows each),
// forward: 17.2 ms in k_solve_cta<1>, 10.5 ms so; without such worlds the launch takes 2 us.
__global__ void __launch_bounds__(128, 4) k_solve_generic_rows(const __grid_constant__ MjbModel m, const __grid_constant__ MjbData d, int smem_per_warp, int min_rows,
                                                              int ordered) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5, wib = threadIdx.x >> 5;
  for (int idx = blockIdx.x * warps + wib; idx < d.nworld; idx += gridDim.x * warps) {
    const int w = ordered ? d.world_order[idx] : idx;
    if (d.world_nefc[w] <= min_rows) {
      if (ordered) break;
      continue;
    }
    solve_generic(m, d, w, lane, d.efc_h + W(w, m.nv * m.nv), smem + size_t(wib) * smem_per_warp, true);
  }
}

void launch_solver_many_rows(const MjbModel* m, const MjbData* d, int min_rows, cudaStream_t s) {
  const int spw = generic_nz_floats(m->nv);
  const size_t bytes = size_t(spw) * kDefaultWarps * sizeof(float);
  static size_t conf[kSmemDevices];
  allow_smem(k_solve_generic_rows, bytes, conf);
  const int ctas = resident_ctas(k_solve_generic_rows, 32 * kDefaultWarps, bytes);
  k_solve_generic_rows<<<std::min(ctas, grid_for(d->nworld, kDefaultWarps)), 32 * kDefaultWarps, bytes, s>>>(
      *m, *d, spw, min_rows, scheduled(d));
}

void launch_solver_generic(const MjbModel* m, const MjbData* d, int warps, cudaStream_t s) {
  if (!scheduled(d)) return launch_solver_many_rows(m, d, -1, s);
  const int spw = generic_nz_floats(m->nv);
  const size_t bytes = size_t(spw) * warps * sizeof(float);
  static size_t conf[kSmemDevices];
  allow_smem(k_solve_generic_queue, size_t(spw) * kDefaultWarps * sizeof(float), conf);
  const int ctas = resident_ctas(k_solve_generic_queue, 32 * warps, bytes);  // ordered in phase 0
  k_solve_generic_queue<<<std::min(ctas, grid_for(d->nworld, warps)), 32 * warps, bytes, s>>>(*m, *d, spw);
}

}  // namespace mjb
