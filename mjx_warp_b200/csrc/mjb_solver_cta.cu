// The FP32 CTA-per-world solver.
#include "mjb_solver_cta_launch.cuh"

namespace mjb {

void launch_solver_cta(const MjbModel* m, const MjbData* d, int nw, int tc, cudaStream_t s) {
  if (nw == 1) {
    launch_solver_many_rows(m, d, SparseFor<1>::kRows, s);  // k_solve_cta<1> leaves those out
    launch_cta<1, false>(m, d, tc, s);
  } else if (nw == 2) launch_cta<2, false>(m, d, tc, s);
  else if (nw == 4) launch_cta<4, false>(m, d, tc, s);
  else if (nw == 16) launch_cta<16, false>(m, d, tc, s);
  else launch_cta<8, false>(m, d, tc, s);
}

bool solver_cta_takes_warp(const MjbModel* m) { return sparse_launch<1>(*m, false); }

}  // namespace mjb
