// Host side of the kernel launches, shared by the library's translation units.  The solvers, the
// single form and the adjoint are units of their own: a stage's routine with one caller in its module
// is inlined and held to that kernel's registers, with several it is compiled apart (8192 and 32768
// humanoid worlds, one module before, split after: k_solve_queue 208 -> 190 and 1300 -> 1216 us,
// k_integrate 67 -> 64 and 236 -> 219, narrowphase 36 -> 28 and 90 -> 59).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "../../include/mjb200.h"

namespace mjb {

constexpr int kSmemDevices = 64;
constexpr int kDefaultWarps = 4;
// dynamic shared memory a CTA of kDefaultWarps warps may use (the opt-in limit of sm_100)
constexpr size_t kMaxSmemPerCta = 227 * 1024;

inline int grid_for(int nworld, int warps) { return (nworld + warps - 1) / warps; }

inline int finish() {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MJB_OK : MJB_ERR_LAUNCH;
}

// opts a kernel in to more than 48 KB of dynamic shared memory (once per kernel, device and size)
template <typename K>
void allow_smem(K kernel, size_t bytes, size_t (&configured)[kSmemDevices]) {
  if (bytes <= 48 * 1024) return;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= kSmemDevices || bytes > configured[dev]) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
    if (dev >= 0 && dev < kSmemDevices) configured[dev] = bytes;
  }
}

// CTAs of `kernel` resident on the whole GPU at once for blocks of `threads` threads and `smem`
// bytes, queried once per (device, kernel, block size, shared-memory size)
template <typename K>
int resident_ctas(K kernel, int threads, size_t smem) {
  struct Entry {
    int dev;
    const void* fn;
    int threads;
    size_t smem;
    int ctas;
  };
  static Entry cache[64];
  static int used = 0;
  static std::mutex mu;
  int dev = 0;
  cudaGetDevice(&dev);
  const void* fn = reinterpret_cast<const void*>(kernel);
  std::lock_guard<std::mutex> lock(mu);
  for (int i = 0; i < used; i++)
    if (cache[i].dev == dev && cache[i].fn == fn && cache[i].threads == threads &&
        cache[i].smem == smem)
      return cache[i].ctas;
  int sms = 0, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  const int n = std::max(1, sms * std::max(1, per_sm));
  if (used < 64) cache[used++] = Entry{dev, fn, threads, smem, n};
  return n;
}

// the Data has the arrays of k_order_worlds' schedule
inline bool scheduled(const MjbData* d) { return d->world_order && d->work_queue && d->world_nefc; }

// the one-warp-per-world solvers for nv <= 32 and a dense mass matrix, spw floats of shared memory per warp: the chosen form's persistent
// one of FP32 FMAs at 5 CTAs per SM (mjb_solver_queue.cu); at 4, the default, or with the Hessian on the
// tensor pipe (mjb_solver_alt.cu); the precision form's (mjb_solver_prec.cu); the plain form's (mjb_solver_plain.cu)
void launch_solver_warp(const MjbModel* m, const MjbData* d, int warps, int spw, cudaStream_t s);
void launch_solver_warp_alt(const MjbModel* m, const MjbData* d, bool tc, int warps, int spw, cudaStream_t s);
void launch_solver_warp_prec(const MjbModel* m, const MjbData* d, int warps, int spw, cudaStream_t s);
// the generic solver for the other models, and for the worlds of more than min_rows rows
// (mjb_solver_generic.cu)
void launch_solver_generic(const MjbModel* m, const MjbData* d, int warps, cudaStream_t s);
void launch_solver_many_rows(const MjbModel* m, const MjbData* d, int min_rows, cudaStream_t s);
int launch_solver_plain(const MjbModel* m, const MjbData* d, cudaStream_t s);
// mjb_step_fused.cu: the single form
void launch_step_fused(const MjbModel* m, const MjbData* d, int integrate, int warps, int spw, size_t smem, cudaStream_t s);
// mjb_step_vjp.cu: the adjoint
int run_step_vjp(const MjbModel* m, const MjbData* d, const float* lam, const float* qvel_prev,
                 float* grad_ctrl, float* grad_qvel, float* grad_qpos, cudaStream_t s);
// the solver of models with nv > 32, nw = 2, 4, 8 or 16 warps per world: FP32 (mjb_solver_cta.cu; also
// nw = 1 where solver_cta_takes_warp; tc: the Hessian on the tensor pipe) and the precision form's
// (mjb_solver_cta_prec.cu; solver_cta_prec_smem: the bytes of shared memory it needs at 16 warps)
void launch_solver_cta(const MjbModel* m, const MjbData* d, int nw, int tc, cudaStream_t s);
bool solver_cta_takes_warp(const MjbModel* m);
void launch_solver_cta_prec(const MjbModel* m, const MjbData* d, int nw, cudaStream_t s);
size_t solver_cta_prec_smem(int nv);

}  // namespace mjb
