// The adjoint of one step (mjb_adjoint.cuh, mjb_deriv.cuh).
#include "mjb_deriv.cuh"
#include "mjb_launch.cuh"

namespace mjb {

// one warp per world; per_warp floats of dynamic shared memory per warp (step_vjp_floats)
__global__ void __launch_bounds__(128) k_step_vjp(const __grid_constant__ MjbModel m, const __grid_constant__ MjbData d,
                                                  const float* lam, const float* qvel_prev,
                                                  float* grad_ctrl, float* grad_qvel,
                                                  float* grad_qpos, int per_warp) {
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= d.nworld) return;
  step_vjp_world(m, d, w, lane, lam, qvel_prev, grad_ctrl, grad_qvel, grad_qpos,
                 smem + size_t(threadIdx.x >> 5) * per_warp);
}

int run_step_vjp(const MjbModel* m, const MjbData* d, const float* lam, const float* qvel_prev,
                 float* grad_ctrl, float* grad_qvel, float* grad_qpos, cudaStream_t s) {
  const int per_warp = (step_vjp_floats(*m, grad_qvel != nullptr, grad_qpos != nullptr) + 3) & ~3;
  const size_t warp_bytes = size_t(per_warp) * sizeof(float);
  int warps = 4;
  while (warps > 1 && warps * warp_bytes > 48 * 1024) warps >>= 1;
  const size_t bytes = warps * warp_bytes;
  if (bytes > 227 * 1024) return MJB_ERR_SCRATCH;
  if (bytes > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_step_vjp, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         int(bytes));
    if (e != cudaSuccess) return MJB_ERR_LAUNCH;
  }
  k_step_vjp<<<grid_for(d->nworld, warps), 32 * warps, bytes, s>>>(
      *m, *d, lam, qvel_prev, grad_ctrl, grad_qvel, grad_qpos, per_warp);
  return finish();
}

}  // namespace mjb
