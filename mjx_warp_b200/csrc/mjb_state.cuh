// Per-world checks and copies that several launch forms share.
#pragma once

#include "mjb_world.cuh"

namespace mjb {

// NaN / Inf check of the integrated state (sets MJB_WS_NONFINITE)
static __device__ void check_finite(const MjbModel& m, const MjbData& d, int w, int lane) {
  bool bad = false;
  for (int i = lane; i < m.nq; i += 32) bad |= !isfinite(d.qpos[W(w, m.nq) + i]);
  for (int i = lane; i < m.nv; i += 32) {
    bad |= !isfinite(d.qvel[W(w, m.nv) + i]);
    bad |= !isfinite(d.qacc[W(w, m.nv) + i]);
  }
  if (__any_sync(WARP_FULL, bad) && lane == 0 && d.world_status) atomicOr(d.world_status + w, MJB_WS_NONFINITE);
}

__device__ __forceinline__ void copy_qacc_smooth(const MjbModel& m, const MjbData& d, int w, int lane) {
  for (int i = lane; i < m.nv; i += 32) d.qacc[W(w, m.nv) + i] = d.qacc_smooth[W(w, m.nv) + i];
  __syncwarp();
}

}  // namespace mjb
