"""Kernel paths chosen by size or alignment, at their edges: rows per world around the small solver's
staged capacity, tree blocks packed four to a tile, constraint rows past eight contacts, and the
one-launch copies of step_io."""

import numpy as np
import pytest
import torch

import mjx_warp_b200 as mjw
from mjx_warp_b200.types import MJ_JAC_DENSE
from helpers import dev, device_data, humanoid, humanoid_state, load, oracle, world_rows
from test_gpu_configs import bin_state, humanoid_spheres_state

pytestmark = pytest.mark.gpu


def corner_xml(nbox):
  """nbox free boxes in a corner of three planes: up to 48 contact rows each."""
  body = '<body pos="0 0 0"><freejoint/><geom type="box" size="0.1 0.08 0.06"/></body>'
  planes = "".join(f'<geom type="plane" zaxis="{z}" size="0 0 1"/>' for z in ("0 0 1", "1 0 0", "0 1 0"))
  return ('<mujoco><option timestep="0.002" iterations="30" ls_iterations="20"/><worldbody>' + planes
          + body * nbox + "</worldbody></mujoco>")


@pytest.mark.parametrize("nbox", [2, 3, 5])
def test_small_solver_rows_per_world(nbox):
  """nv = 12 and 18 stage up to 64 rows per world (two per lane past 32), nv = 30 only 32: worlds of
  0 to over 64 rows.  The solver's cost, evaluated in FP64 on the device's rows, is the minimum that
  an FP64 Newton iteration finds, within the FP32 evaluation of a cost of n rows (2^-24 a term) and
  the solver's own stopping tolerance."""
  mjm = load(corner_xml(nbox))
  nworld, rng = 48, np.random.default_rng(nbox)
  q = np.tile(mjm.qpos0, (nworld, 1))
  x = q.reshape(nworld, nbox, 7)
  x[:, :, :3] = rng.uniform(0.02, 0.5, (nworld, nbox, 3)) * (1.0 - np.arange(nworld)[:, None, None] / nworld) + 0.02
  r = rng.normal(size=(nworld, nbox, 4))
  x[:, :, 3:] = r / np.linalg.norm(r, axis=2, keepdims=True)
  m = mjw.put_model(mjm)
  d = device_data(mjm, q, rng.normal(0.0, 0.1, (nworld, mjm.nv)), np.zeros((nworld, 0)),
                  nconmax=64 * nworld, njmax=256 * nworld)
  mjw.forward(m, d)
  torch.cuda.synchronize()
  assert np.all(mjw.world_status(d) == 0)
  n, idx = world_rows(d, "efc")
  assert n.min() <= 32 < n.max() and (nbox == 2 or n.max() > 64)
  J, D, aref = (t.cpu().numpy().astype(np.float64) for t in (d.efc.J, d.efc.D, d.efc.aref))
  M, f, qacc = dev(d.qM).reshape(nworld, mjm.nv, mjm.nv), dev(d.qfrc_smooth), dev(d.qacc)
  at = 0
  for w in range(nworld):
    rows = idx[at:at + n[w]]
    at += n[w]
    Jw, Dw, aw, smooth = J[rows], D[rows], aref[rows], np.linalg.solve(M[w], f[w])

    def cost(a):
      e = np.minimum(Jw @ a - aw, 0.0)
      return 0.5 * (a - smooth) @ M[w] @ (a - smooth) + 0.5 * np.sum(Dw * e * e)

    a = smooth.copy()
    for _ in range(200):  # damped Newton
      e = np.minimum(Jw @ a - aw, 0.0)
      g = M[w] @ (a - smooth) + Jw.T @ (Dw * e)
      step = np.linalg.solve(M[w] + Jw[e < 0].T @ (Dw[e < 0, None] * Jw[e < 0]), -g)
      t = 1.0
      while cost(a + t * step) > cost(a) and t > 1e-9:
        t *= 0.5
      a = a + t * step
    c, best = cost(qacc[w]), cost(a)
    tol = (n[w] + mjm.nv) * 2.0 ** -24 * 10 * best + mjm.opt.tolerance * mjm.stat.meaninertia * mjm.nv * 10
    assert c <= best + max(tol, 1e-4 * best), (w, n[w], c, best)
