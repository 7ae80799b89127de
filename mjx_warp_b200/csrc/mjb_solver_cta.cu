// The FP32 CTA-per-world solver.
#include "mjb_solver_cta_launch.cuh"

namespace mjb {

// The worlds of more rows than the one-warp structure holds, by the generic solver, beside
// k_solve_cta<1>, which leaves them out: there a world takes 24 KB of shared memory, so nine warps run on
// an SM, here twenty.  In k_order_worlds' order those worlds come first (the buckets of its sort hold up to
// 254 rows apart), so every warp stops at its first smaller one.  2048 worlds of 20 boxes lying on a plane
// (320 rows each), forward: 17.2 ms in k_solve_cta<1>, 11.7 ms so; without such worlds the launch takes 2 us.
__global__ void __launch_bounds__(128, 5) k_solve_many_rows(const __grid_constant__ MjbModel m, const __grid_constant__ MjbData d, int smem_per_warp) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5, wib = threadIdx.x >> 5;
  const bool ordered = d.work_queue != nullptr;
  for (int idx = blockIdx.x * warps + wib; idx < d.nworld; idx += gridDim.x * warps) {
    const int w = ordered ? d.world_order[idx] : idx;
    if (d.world_nefc[w] <= SparseFor<1>::kRows) {
      if (ordered) break;
      continue;
    }
    solve_generic(m, d, w, lane, d.efc_h + W(w, m.nv * m.nv), smem + size_t(wib) * smem_per_warp, true);
  }
}

static void launch_many_rows(const MjbModel* m, const MjbData* d, cudaStream_t s) {
  const int spw = generic_nz_floats(m->nv);
  const size_t bytes = size_t(spw) * kDefaultWarps * sizeof(float);  // 18 KB
  MjbData dd = *d;
  if (!(d->world_order && d->world_nefc)) dd.work_queue = nullptr;
  const int ctas = resident_ctas(k_solve_many_rows, 32 * kDefaultWarps, bytes);
  k_solve_many_rows<<<std::min(ctas, grid_for(d->nworld, kDefaultWarps)), 32 * kDefaultWarps, bytes, s>>>(*m, dd, spw);
}

void launch_solver_cta(const MjbModel* m, const MjbData* d, int nw, int tc, cudaStream_t s) {
  if (nw == 1) {
    launch_many_rows(m, d, s);
    launch_cta<1, false>(m, d, tc, s);
  } else if (nw == 2) launch_cta<2, false>(m, d, tc, s);
  else if (nw == 4) launch_cta<4, false>(m, d, tc, s);
  else if (nw == 16) launch_cta<16, false>(m, d, tc, s);
  else launch_cta<8, false>(m, d, tc, s);
}

bool solver_cta_takes_warp(const MjbModel* m) { return sparse_launch<1>(*m, false); }

}  // namespace mjb
