"""The solver of models of several kinematic trees (nv > 32) over nonzero trees and tiles only, at the
edges of its structure: 2 to 65 trees (64 is the most that it takes), tree sizes 6 and 27, matrices
whose last 32-dof panel is partial, worlds without rows, rows and tree pairs past its capacities."""

import json

import numpy as np
import pytest
import torch

import mjx_warp_b200 as mjw
from mjx_warp_b200.types import MJ_JAC_DENSE, MJ_JAC_SPARSE
from oracle import Oracle
from helpers import dev, device_data, load, world_rows
from test_gpu_configs import bin_state, humanoid_spheres_state

pytestmark = pytest.mark.gpu


def spheres_xml(n):
  """n free spheres on a grid over a plane, every other one touching it."""
  bodies = "\n".join(
    f'<body pos="{0.3 * (i % 9):.2f} {0.3 * (i // 9):.2f} {0.095 if i % 2 else 0.5}"><freejoint/>'
    f'<geom type="sphere" size="0.1"/></body>' for i in range(n))
  return ('<mujoco><option timestep="0.002"/><worldbody><geom type="plane" size="0 0 1"/>'
          + bodies + "</worldbody></mujoco>")


def chain_xml(n):
  """One tree: a chain of n hinges whose links touch the plane below them only."""
  s = '<mujoco><option timestep="0.002"/><worldbody><geom type="plane" size="0 0 1" pos="0 0 -0.1"/>'
  for i in range(n):
    s += (f'<body pos="{0.1 if i else 0} 0 0"><joint type="hinge" damping="0.3" axis="{i % 2} {(i + 1) % 2} 0.2"/>'
          '<geom type="capsule" fromto="0 0 0 0.1 0 0" size="0.02" contype="0" conaffinity="1"/>')
  return s + "</body>" * n + "</worldbody></mujoco>"


def star_xml(n, dofs):
  """n trees resting on one long capsule, the first tree, whose elimination couples them all: free
  capsules, each with dofs - 6 hinges hanging from it."""
  s = ('<mujoco><option timestep="0.002"/><worldbody><body pos="0 0 1"><freejoint/>'
       f'<geom type="capsule" fromto="0 0 0 {0.5 * n:g} 0 0" size="0.1"/></body>')
  for i in range(n):
    s += (f'<body pos="{0.25 + 0.5 * i} 0 1.19"><freejoint/>'
          '<geom type="capsule" fromto="0 -0.1 0 0 0.1 0" size="0.1"/>')
    for k in range(dofs - 6):
      s += (f'<body pos="0 0 0.05"><joint type="hinge" damping="0.3" axis="{k % 2} {(k + 1) % 2} 0.2"/>'
            '<geom type="capsule" fromto="0 0 0 0 0 0.05" size="0.02" contype="0" conaffinity="0"/>')
    s += "</body>" * (dofs - 5)
  return s + "</worldbody></mujoco>"


def case(name):
  """(model, qpos, qvel, ctrl, rows capacity per world)"""
  opt = dict(iterations=0, ls_iterations=10, jacobian=MJ_JAC_DENSE)
  if name.startswith("spheres"):
    mjm = load(spheres_xml(int(name[7:])), **opt)
    rng = np.random.default_rng(1)
    q = np.tile(mjm.qpos0, (5, 1))
    x = q.reshape(5, -1, 7)
    x[:, :, :2] += rng.uniform(-0.12, 0.12, x[:, :, :2].shape)
    x[0, :, 2] += 5.0  # a world without rows
    return mjm, q, rng.normal(0.0, 0.1, (5, mjm.nv)), np.zeros((5, 0)), 512
  if name.startswith("star"):
    mjm = load(star_xml(*(int(n) for n in name[4:].split("x"))), **opt)
    rng = np.random.default_rng(8)
    q = np.tile(mjm.qpos0, (3, 1))
    q[1, 2] -= 0.5  # a world whose trees do not touch
    return mjm, q, rng.normal(0.0, 0.01, (3, mjm.nv)), np.zeros((3, 0)), 256
  if name == "humanoid_spheres":
    mjm = load("humanoid_spheres.xml", **opt)
    q, v, u, _ = humanoid_spheres_state(mjm, load("humanoid.xml"), 8, seed=3)
    return mjm, q, v, u, 384
  mjm = load("bin.xml", **opt)
  q, v, u = bin_state(mjm, 4, seed=3 if name == "bin_pairs" else 6)
  x = q.reshape(4, -1, 7)
  if name == "bin_rows":  # every body in one heap in worlds 0 and 1
    x[:2, :, :3] = np.array([0.0, 0.0, 0.3]) + 0.28 * (x[:2, :, :3] - np.array([0.0, 0.0, 0.19]))
  if name == "bin_pairs":  # heaps of 477 to 624 tree pairs
    x[:, :, :3] = np.array([0.0, 0.0, 0.3]) + 0.5 * (x[:, :, :3] - np.array([0.0, 0.0, 0.19]))
  return mjm, q, v, u, 2048


def tree_pairs(mjm, J):
  """Nonzero tree pairs of the factor of H for the rows J: each tree with itself, with the trees that
  a row couples it with, and the fill of eliminating the trees in dof order."""
  tree = np.asarray(mjm.dof_bodyid)
  tree = np.unique(np.asarray(mjm.body_rootid)[tree], return_inverse=True)[1]
  n = tree.max() + 1
  touch = np.zeros((len(J), n), dtype=np.int64)
  np.maximum.at(touch.T, tree, (J != 0).T.astype(np.int64))
  C = (touch.T @ touch > 0) | np.eye(n, dtype=bool)
  for k in range(n):
    later = np.nonzero(C[k + 1:, k])[0] + k + 1
    C[np.ix_(later, later)] = True
  return int(np.tril(C).sum())


@pytest.mark.parametrize("warps", [2, 4])
@pytest.mark.parametrize("name", ["spheres6", "spheres11", "spheres64", "spheres65", "humanoid_spheres",
                                  "bin", "bin_rows", "bin_pairs", "star20x22", "star29x17"])
def test_factor_of_the_hessian(name, warps):
  """Also past the lists of a panel's updated tiles (20 coupled trees of 22 dofs) and of its rows below (29 of
  17), with few rows.  With no iterations efc_h is the factor of H = qM + J_a' D_a J_a at the warmstart's active set:
  zero where H's factor is, and L L' = H within the backward error of an FP32 Cholesky factorisation
  (nv + 1 roundings of 2^-24 per entry, doubled for the assembly)."""
  mjm, q, v, u, cap = case(name)
  nworld = q.shape[0]
  m = mjw.put_model(mjm)
  d = device_data(mjm, q, v, u, nconmax=800 * nworld, njmax=cap * nworld)
  try:
    mjw.set_tune(m, d, solver_cta_warps=warps)
    mjw.forward(m, d)
    torch.cuda.synchronize()
  finally:
    mjw.set_tune(m, d, solver_cta_warps=4 if mjm.nv > 128 else 0)
  assert np.all(mjw.world_status(d) == 0)
  n, idx = world_rows(d, "efc")
  if name == "bin_rows":
    assert n.max() > 736 > n.min()
  J, D = (x.cpu().numpy().astype(np.float64) for x in (d.efc.J, d.efc.D))
  act = d.efc.active.cpu().numpy().astype(bool)
  if name == "bin_pairs":  # more pairs than the structure's 512 with no more than its 736 rows, and fewer
    first = np.cumsum(n) - n
    pairs = np.array([tree_pairs(mjm, J[idx[a:a + k]]) for a, k in zip(first, n)])
    assert np.any((pairs > 512) & (n <= 736)) and np.any((pairs <= 512) & (n <= 736)), (pairs, n)
  at = 0
  for w in range(nworld):
    rows = idx[at:at + n[w]]
    at += n[w]
    rows = rows[act[rows]]
    H = d.qM[w].cpu().numpy().astype(np.float64) + J[rows].T @ (D[rows, None] * J[rows])
    L = np.tril(d.efc.h[w].cpu().numpy().astype(np.float64))
    r = np.linalg.norm(L @ L.T - H) / np.linalg.norm(H)
    assert r < 2 * (mjm.nv + 1) * 2.0 ** -24, (w, r)


@pytest.mark.parametrize("name", ["spheres6", "spheres11", "spheres16", "humanoid_spheres", "star8x6", "star18x6"])
def test_one_warp_form_equals_plain(name):
  """Up to 128 dofs the chosen form solves a world by one warp over the nonzero trees in the plain
  form's arithmetic: equal values, whether the world fits the structure or (more than 192 rows: the
  16 spheres in one heap; more than three quarters of the tree pairs nonzero, or more of them than it
  holds: 8 and 18 capsules on one) takes the generic solver."""
  mjm, q, v, u, cap = case(name)
  mjm.opt.iterations = 10
  if name == "spheres16":
    x = q.reshape(5, -1, 7)
    x[1:3, :, :3] = 0.15 + 0.05 * (x[1:3, :, :3] - x[1:3, :1, :3])
  nworld = q.shape[0]
  m = mjw.put_model(mjm)
  out = {}
  for form in (1, 0):
    d = device_data(mjm, q, v, u, nconmax=800 * nworld, njmax=cap * nworld)
    mjw.forward(m, d, fused=form)
    torch.cuda.synchronize()
    assert np.all(mjw.world_status(d) == 0)
    out[form] = d
  n = world_rows(out[1], "efc")[0]
  assert name != "spheres16" or n.max() > 192 > n.min()
  if name == "star18x6":
    idx = world_rows(out[1], "efc")[1]
    J = out[1].efc.J.cpu().numpy()
    assert n[0] <= 192 and tree_pairs(mjm, J[idx[:n[0]]]) > 160
  for f in ("qacc", "qfrc_constraint"):
    assert torch.equal(getattr(out[1], f), getattr(out[0], f)), f
  for f in ("cost", "Ma", "h"):
    a, b = getattr(out[1].efc, f), getattr(out[0].efc, f)
    assert torch.equal(a.tril(), b.tril()) if f == "h" else torch.equal(a, b), f


@pytest.mark.parametrize("name", ["spheres6", "spheres66", "bin"])
def test_rows_and_hessian_at_any_address(name):
  """efc.J and efc.h as contiguous views at a 4-byte offset give what 16-byte aligned ones give: the
  one-warp form (6 spheres), the dense one (66 trees, nv a multiple of 4) and the sparse one."""
  mjm, q, v, u, cap = case(name)
  mjm.opt.iterations = 10
  nworld = q.shape[0]
  m = mjw.put_model(mjm)
  out = []
  for offset in (0, 1):
    d = device_data(mjm, q, v, u, nconmax=800 * nworld, njmax=cap * nworld)
    for f in ("J", "h"):
      t = getattr(d.efc, f)
      base = torch.zeros(t.numel() + 4, device="cuda")
      setattr(d.efc, f, base[offset:offset + t.numel()].view(t.shape))
      assert getattr(d.efc, f).data_ptr() % 16 == 4 * offset
    mjw.forward(m, d)
    torch.cuda.synchronize()
    assert np.all(mjw.world_status(d) == 0)
    out.append((d.efc.J.cpu()[world_rows(d, "efc")[1]], d.efc.h.cpu().tril(), d.qacc.cpu()))
  for a, b in zip(*out):
    assert torch.equal(a, b)


@pytest.mark.parametrize("name, tc", [("chain40", False), ("spheres66", False), ("spheres11", True)])
def test_dense_launches_keep_their_shared_memory(name, tc, tmp_path):
  """One tree, more than 64 trees and the tensor-core assembly do not look for a structure: their launch
  asks for the dense form's shared memory only, and eight two-warp blocks fit on an SM (228 KB, 1 KB of
  each block's reserved)."""
  if name.startswith("chain"):
    mjm = load(chain_xml(int(name[5:])), jacobian=MJ_JAC_DENSE)
    q, v, u = np.tile(mjm.qpos0, (5, 1)), np.zeros((5, mjm.nv)), np.zeros((5, 0))
    q += np.random.default_rng(2).uniform(-0.3, 0.3, q.shape)
  else:
    mjm, q, v, u, _ = case(name)
  m = mjw.put_model(mjm)
  d = device_data(mjm, q, v, u, nconmax=5 * 128, njmax=5 * 512)
  try:
    mjw.set_tune(m, d, solver_cta_warps=2, hessian_tc=tc)
    mjw.forward(m, d)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
      mjw.forward(m, d)
      torch.cuda.synchronize()
  finally:
    mjw.set_tune(m, d, solver_cta_warps=4 if mjm.nv > 128 else 0)
  assert np.all(mjw.world_status(d) == 0)
  p.export_chrome_trace(str(tmp_path / "trace.json"))
  events = json.loads((tmp_path / "trace.json").read_text())["traceEvents"]
  smem = [e["args"]["shared memory"] for e in events if "k_solve_cta" in e.get("name", "") and "shared memory" in e.get("args", {})]
  assert smem and max(smem) <= 228 * 1024 // 8 - 1024, smem


@pytest.mark.parametrize("ordered", [True, False])
def test_one_warp_worlds_past_the_row_capacity(ordered):
  """Worlds of 0 to 320 rows (boxes on a plane, 4 contacts each) mixed in one batch, more and fewer than the
  192 rows of the one-warp structure: every world is solved, once, to the plain form's values, with the
  work queue and without."""
  boxes = "".join(f'<body pos="{0.5 * (i % 5)} {0.5 * (i // 5)} 0.058"><freejoint/>'
                  '<geom type="box" size="0.1 0.08 0.06"/></body>' for i in range(20))
  mjm = load('<mujoco><option timestep="0.002"/><worldbody><geom type="plane" size="0 0 1"/>' + boxes
             + "</worldbody></mujoco>", iterations=5, ls_iterations=10, jacobian=MJ_JAC_DENSE)
  nworld, rng = 37, np.random.default_rng(4)
  q = np.tile(mjm.qpos0, (nworld, 1))
  x = q.reshape(nworld, 20, 7)
  x[:, :, :2] += rng.uniform(-0.05, 0.05, (nworld, 20, 2))
  for w in range(nworld):
    x[w, w % 21:, 2] += 1.0  # w mod 21 boxes touch the plane
  v = rng.normal(0.0, 0.1, (nworld, mjm.nv))
  m = mjw.put_model(mjm)
  out = {}
  for form in (1, 0):
    d = device_data(mjm, q, v, np.zeros((nworld, 0)), nconmax=100 * nworld, njmax=400 * nworld)
    if not ordered:
      d.work_queue = None
    mjw.forward(m, d, fused=form)
    torch.cuda.synchronize()
    assert np.all(mjw.world_status(d) == 0)
    out[form] = d
  n = world_rows(out[1], "efc")[0]
  assert n.min() == 0 and n.max() == 320 and np.any(n == 192) and np.any(n == 208)
  for f in ("qacc", "qfrc_constraint", "qacc_warmstart"):
    assert torch.equal(getattr(out[1], f), getattr(out[0], f)), f
  assert torch.equal(out[1].efc.h.tril(), out[0].efc.h.tril())


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("name", ["spheres6", "spheres11", "bin"])
def test_nonfinite_force_reaches_every_tree(name, bad):
  """A NaN or an infinite force on one dof of one tree: the world's accelerations are not finite where the
  plain form's are not (its dense solve multiplies them with the zeros between the trees), and the
  other worlds are what they are without it."""
  mjm, q, v, u, cap = case(name)
  mjm.opt.iterations = 5
  nworld = q.shape[0]
  m = mjw.put_model(mjm)
  qacc = {}
  for key, form, force in (("clean", 1, 0.0), ("chosen", 1, bad), ("plain", 0, bad)):
    d = device_data(mjm, q, v, u, nconmax=800 * nworld, njmax=cap * nworld)
    d.qfrc_applied[1, 8] = force
    mjw.forward(m, d, fused=form)
    torch.cuda.synchronize()
    qacc[key] = dev(d.qacc)
  plain = np.isfinite(qacc["plain"])
  assert not plain[1].any() and np.delete(plain, 1, axis=0).all()
  assert np.array_equal(np.isfinite(qacc["chosen"]), plain)
  assert np.array_equal(np.delete(qacc["chosen"], 1, axis=0), np.delete(qacc["clean"], 1, axis=0))


@pytest.mark.parametrize("jacobian", [MJ_JAC_DENSE, MJ_JAC_SPARSE])
@pytest.mark.parametrize("solver, iterations, ls_iterations, ls_parallel",
                         [(2, 20, 20, False), (2, 20, 50, True), (1, 100, 20, False), (1, 100, 50, True)])
@pytest.mark.parametrize("name", ["spheres11", "humanoid_spheres", "bin"])
def test_solvers_and_searches_over_trees(name, solver, iterations, ls_iterations, ls_parallel, jacobian):
  """Newton and CG, the iterative and the parallel search, dense and sparse mass matrix, one warp (66 and 123
  dofs) and four warps (384): the cost is the oracle's, by the reference's acceptance (solver_test.py:
  2.5 % above it at most)."""
  mjm, q, v, u, cap = case(name)
  mjm.opt.solver, mjm.opt.iterations, mjm.opt.ls_iterations, mjm.opt.jacobian = solver, iterations, ls_iterations, jacobian
  nworld = q.shape[0]
  m = mjw.put_model(mjm)
  m.opt.ls_parallel = ls_parallel
  d = device_data(mjm, q, v, u, nconmax=800 * nworld, njmax=cap * nworld)
  mjw.forward(m, d)
  torch.cuda.synchronize()
  assert m.opt.is_sparse == (jacobian == MJ_JAC_SPARSE) and np.all(mjw.world_status(d) == 0)
  o = Oracle(mjm, nworld, 64, ls_parallel=ls_parallel)
  for f, x in (("qpos", q), ("qvel", v), ("ctrl", u)):
    if x.shape[1]:
      o.set(f, x)
  o.run("forward", nthreads=8)
  np.testing.assert_array_equal(world_rows(d, "efc")[0], o.rows("efc_D")[0])
  cost, ref = d.efc.cost.cpu().numpy(), o.scalar("cost")
  assert np.all(cost <= ref + 0.025 * np.abs(ref) + 1e-3), (cost, ref)
