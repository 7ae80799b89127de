// The precision form's CTA-per-world solver.
#include "mjb_solver_cta_launch.cuh"

namespace mjb {

void launch_solver_cta_prec(const MjbModel* m, const MjbData* d, int nw, cudaStream_t s) {
  if (nw == 2) launch_cta<2, true>(m, d, 0, s);
  else if (nw == 4) launch_cta<4, true>(m, d, 0, s);
  else if (nw == 16) launch_cta<16, true>(m, d, 0, s);
  else launch_cta<8, true>(m, d, 0, s);
}

size_t solver_cta_prec_smem(int nv) { return size_t(cta_solver_smem_floats(nv, 16, true, false)) * sizeof(float); }

}  // namespace mjb
