"""Kernel paths chosen by size or alignment, at their edges: rows per world around the small solver's
staged capacity, tree blocks packed four to a tile, constraint rows past eight contacts, and the
one-launch copies of step_io."""

import ctypes

import numpy as np
import pytest
import torch

import mjx_warp_b200 as mjw
from mjx_warp_b200 import _abi
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
  an FP64 Newton iteration finds, within 1e-4 of it (the line search stops within its own tolerance of a
  step's minimum) or, where that is more, the FP32 evaluation of a cost of n rows (2^-24 a term) and the
  solver's stopping tolerance."""
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


def spheres_xml(sizes):
  """Trees of the given numbers of slide / hinge dofs (6: a free sphere)."""
  out = []
  for i, s in enumerate(sizes):
    if s == 6:
      out.append(f'<body pos="{i} 0 1"><freejoint/><geom type="sphere" size="0.1"/></body>')
      continue
    chain, close = "", ""
    for k in range(s):
      chain += (f'<body pos="{i if k == 0 else 0} 0 {1 if k == 0 else -0.1}"><joint type="hinge" damping="0.3" axis="{k % 2} {(k + 1) % 2} 0.2"/>'
                '<geom type="capsule" fromto="0 0 0 0.02 0 -0.1" size="0.02"/>')
      close += "</body>"
    out.append(chain + close)
  return ('<mujoco><option timestep="0.002"><flag contact="disable"/></option><worldbody>' + "".join(out)
          + "</worldbody></mujoco>")


@pytest.mark.parametrize("form", [1, 3])
@pytest.mark.parametrize("sizes", [(1, 8), (6, 5), (8, 9, 8, 8), (6,) * 6, (8, 1, 7, 6, 2, 27, 6, 6), (33, 6, 6)])
def test_packed_tree_blocks(sizes, form):
  """Factor, solve and damped integration of dense mass matrices of trees of 1 to 33 dofs: runs of
  trees of up to 8 are taken four at a time (nv >= 32 for the factor).  L L' = M within the backward
  error of an FP32 Cholesky factorisation of the largest block; qacc_smooth and the Euler step with implicit damping against
  FP64 solves of the same matrices, within cond(M) roundings."""
  if form == 3 and max(sizes) > 32:
    pytest.skip("the precision form takes trees of up to 32 dofs")
  mjm = load(spheres_xml(sizes), jacobian=MJ_JAC_DENSE)
  nworld, rng = 5, np.random.default_rng(len(sizes))
  q = np.tile(mjm.qpos0, (nworld, 1))
  hinge = np.asarray(mjm.jnt_type) == 3
  q[:, np.asarray(mjm.jnt_qposadr)[hinge]] += rng.uniform(-0.5, 0.5, (nworld, int(hinge.sum())))
  v = rng.normal(0.0, 0.2, (nworld, mjm.nv))
  m = mjw.put_model(mjm)
  d = device_data(mjm, q, v, np.zeros((nworld, 0)), nconmax=8 * nworld, njmax=64 * nworld)
  mjw.step(m, d, fused=form)
  torch.cuda.synchronize()
  nv, h = mjm.nv, mjm.opt.timestep
  M = dev(d.qM).reshape(nworld, nv, nv)
  L = dev(d.qLD).reshape(nworld, nv, nv)
  f, a = dev(d.qfrc_smooth), dev(d.qacc_smooth)
  damp = np.asarray(mjm.dof_damping)
  for w in range(nworld):
    eps = 2.0 ** -24
    assert np.linalg.norm(L[w] @ L[w].T - M[w]) <= 2 * (max(sizes) + 1) * eps * np.linalg.norm(M[w])
    ref = np.linalg.solve(M[w], f[w])
    assert np.linalg.norm(a[w] - ref) <= 4 * max(sizes) * eps * np.linalg.cond(M[w]) * np.linalg.norm(ref)
    Md = M[w] + h * np.diag(damp)
    step = (dev(d.qvel)[w] - v[w].astype(np.float32)) / h
    ref = np.linalg.solve(Md, f[w] + dev(d.qfrc_constraint)[w])
    tol = 4 * max(sizes) * eps * np.linalg.cond(Md) * np.linalg.norm(ref) + 2 * eps * np.linalg.norm(v[w]) / h
    assert np.linalg.norm(step - ref) <= tol, (w, np.linalg.norm(step - ref), tol)


@pytest.mark.parametrize("model", ["humanoid", "humanoid_spheres", "bin"])
def test_constraint_rows_vs_oracle(model):
  """Rows of 1 to 50 contacts per world (scalars formed eight contacts at a time; past 32 dofs only the
  dofs of the two bodies' trees are visited)."""
  if model == "humanoid":
    mjm = humanoid()
    q, v, u = humanoid_state(mjm, 16, seed=5)
  elif model == "bin":
    mjm = load("bin.xml", jacobian=MJ_JAC_DENSE)
    q, v, u = bin_state(mjm, 6, seed=9)
  else:
    mjm = load("humanoid_spheres.xml", jacobian=MJ_JAC_DENSE)
    q, v, u, _ = humanoid_spheres_state(mjm, load("humanoid.xml"), 16, seed=9)
  nworld = q.shape[0]
  m = mjw.put_model(mjm)
  d = device_data(mjm, q, v, u, nconmax=600 * nworld, njmax=512 * nworld)
  mjw.forward(m, d)
  o = oracle(mjm, q, v, u, 32)
  o.run("forward_nosolve")
  torch.cuda.synchronize()
  n, idx = world_rows(d, "efc")
  cnt, D = o.rows("efc_D")
  np.testing.assert_array_equal(n, cnt)
  for name, t in (("efc_D", d.efc.D), ("efc_aref", d.efc.aref)):
    got = t.cpu().numpy().astype(np.float64)[idx]
    ref = np.asarray(o.rows(name)[1], dtype=np.float64).reshape(-1)
    # the reference tests' tolerance on constraint rows
    np.testing.assert_allclose(got, ref, rtol=2e-3, atol=2e-3 * max(1.0, np.abs(ref).max() * 1e-3), err_msg=name)
  # J from the device's own contacts and motion axes in FP64 (the frame of two nearly parallel capsules
  # depends on the last bits of their poses), within the roundings of a term of a row
  cn, cidx = world_rows(d, "contact")
  c = {k: getattr(d.contact, k).cpu().numpy()[cidx] for k in ("dist", "pos", "frame", "includemargin", "friction", "geom", "dim")}
  J = d.efc.J.cpu().numpy().astype(np.float64)[idx]
  cdof, com = dev(d.cdof).reshape(nworld, mjm.nv, 6), dev(d.subtree_com).reshape(nworld, mjm.nbody, 3)
  gb, root, par = (np.asarray(x) for x in (mjm.geom_bodyid, mjm.body_rootid, mjm.body_parentid))
  db = np.asarray(mjm.dof_bodyid)
  chain = np.zeros((mjm.nbody, mjm.nv), dtype=bool)
  for b in range(1, mjm.nbody):
    chain[b] = chain[par[b]] | (db == b)
  row = at = 0
  for w in range(nworld):
    act = [k for k in range(at, at + cn[w]) if c["dim"][k] == 3 and c["dist"][k] < c["includemargin"][k]]
    at += cn[w]
    row += n[w] - 4 * len(act)  # the limit rows
    for k in act:
      jac = []
      for g in c["geom"][k]:
        off = c["pos"][k].astype(np.float64) - com[w, root[gb[g]]]
        jac.append((cdof[w, :, 3:] + np.cross(cdof[w, :, :3], off)) * chain[gb[g]][:, None])
      diff = (jac[1] - jac[0]) @ c["frame"][k].astype(np.float64).reshape(3, 3).T
      f = c["friction"][k]
      for e, ref in enumerate((diff[:, 0] + f[0] * diff[:, 1], diff[:, 0] - f[0] * diff[:, 1],
                               diff[:, 0] + f[1] * diff[:, 2], diff[:, 0] - f[1] * diff[:, 2])):
        scale = max(1.0, np.abs(jac[0]).max(), np.abs(jac[1]).max())
        assert np.abs(J[row + e] - ref).max() <= 32 * 2.0 ** -24 * scale * 4, (w, k, e)
      row += 4
  assert row == len(idx)


@pytest.mark.parametrize("offset", [0, 1, 3])
def test_step_io_copies_by_alignment(offset):
  """Inputs and outputs at 4-byte offsets from 16-byte alignment give what aligned ones give."""
  mjm = humanoid()
  q, v, u = humanoid_state(mjm, 7, seed=4)
  m = mjw.put_model(mjm)
  outs = []
  for off in (0, offset):
    d = device_data(mjm, q, v, u)

    def at(shape, src=None):
      n = int(np.prod(shape))
      t = torch.full((n + off + 4,), 7.0, device="cuda")
      view = t[off:off + n].view(shape)
      if src is not None:
        view.copy_(torch.as_tensor(src, dtype=torch.float32))
      return view

    ins = {"qpos": at(q.shape, q), "qvel": at(v.shape, v), "ctrl": at(u.shape, u)}
    out = {"qpos": at(q.shape), "qvel": at(v.shape), "xpos": at((7, mjm.nbody, 3))}
    mjw.step_io(m, d, 2, inputs=ins, outputs=tuple(out), out=out)
    torch.cuda.synchronize()
    outs.append({k: t.clone() for k, t in out.items()})
  for k in outs[0]:
    assert torch.equal(outs[0][k], outs[1][k]), k


def test_step_io_overlapping_buffers_keep_their_order():
  """A copy whose source is another copy's destination: qvel comes from the Data's own warmstart,
  which the next input then replaces."""
  mjm = humanoid()
  q, v, u = humanoid_state(mjm, 5, seed=2)
  m = mjw.put_model(mjm)
  d = device_data(mjm, q, v, u, warmstart=v)
  want = device_data(mjm, q, v, u)
  mjw.step_io(m, d, 1, inputs={"qvel": d.qacc_warmstart, "qacc_warmstart": torch.zeros_like(d.qvel)}, outputs=())
  mjw.step_io(m, want, 1, outputs=())
  torch.cuda.synchronize()
  assert torch.equal(d.qvel, want.qvel)


@pytest.mark.parametrize("field", ["qpos", "qpos_out"])
@pytest.mark.parametrize("pinned", [False, True])
def test_step_io_host_buffers(field, pinned):
  """The C entry takes pinned host buffers and refuses pageable ones (a copy of those would wait for the
  host).  Under capture, so nothing runs."""
  mjm = humanoid()
  q, v, u = humanoid_state(mjm, 4, seed=1)
  m = mjw.put_model(mjm)
  d = device_data(mjm, q, v, u)
  mjw.step(m, d)  # the forked streams exist before the capture
  torch.cuda.synchronize()
  host = torch.zeros(q.shape, dtype=torch.float32, pin_memory=pinned)
  io = _abi.MjbStepIO()
  setattr(io, field, host.data_ptr())
  g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
  with torch.cuda.stream(s):
    g.capture_begin(capture_error_mode="thread_local")
    rc = _abi.lib().mjb_step_io(ctypes.byref(_abi.model_view(m)), ctypes.byref(_abi.data_view(d)),
                                ctypes.byref(io), 1, None, s.cuda_stream)
    g.capture_end()
  _abi.lib().mjb_error_string(rc)  # takes the error back
  assert rc == (0 if pinned else 3)  # MJB_ERR_LAUNCH
