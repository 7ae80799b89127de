"""The workloads that performance of the batched step is measured on.

Each case is one call of the public API as a user's program makes it: `step_io` (the host-framework
step: state and control in, one step, state and observations out; every pass therefore starts from
the same inputs) launched eagerly or replayed from a captured CUDA graph, and a differentiated
rollout (`derivative.Rollout` behind torch.autograd).  Models, solver settings, world counts and
seeded states are those of the benchmark's configurations and of the tests; the solver's iteration
counts are the model files' own, or the benchmark's 3 Newton / 4 line-search iterations.

listed() / draw(rng) give cases, prepare(case, seed) the inputs and the handles a program keeps,
run(state) one pass, work(case) what a pass cannot do without.
"""

import functools
import os

import torch

import mjx_warp_b200 as mjw
from mjx_warp_b200 import mjcf

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# model -> contact and constraint-row capacity per world (as the tests and the benchmark size
# them), the world counts it is run with, and per-world means of its seeded states that work()
# needs: constraint rows, dofs that a row touches, dofs of its kinematic trees
MODELS = {
  "humanoid": dict(nconmax=64, njmax=256, worlds=(1, 32768), rows=9, touched=12, trees=(27,)),
  "sphere_chain": dict(nconmax=16, njmax=64, worlds=(1, 16384), rows=2, touched=5, trees=(6, 5)),
  "humanoid_spheres": dict(nconmax=96, njmax=384, worlds=(16, 4096), rows=9, touched=9,
                           trees=(27,) + (6,) * 16),
  "bin": dict(nconmax=600, njmax=512, worlds=(16, 4096), rows=162, touched=11, trees=(6,) * 64),
}
CHOSEN, PRECISION = 1, 3
EULER, IMPLICITFAST = 0, 3
DENSE, AUTO = 0, 2
FILE, BENCH = 0, 3  # Newton iterations: the model file's, or the benchmark's 3 (4 of line search)
HORIZON, CHECKPOINT = 8, 4  # the differentiated rollout
# what a training or planning loop reads back: the next state, the warmstart it hands to the next
# call, and the observations that MuJoCo's humanoid tasks are built from
OUTPUTS = ("qpos", "qvel", "qacc_warmstart", "xpos", "subtree_com", "cvel")


def _case(name, model, nworld, integrator=EULER, form=CHOSEN, jacobian=DENSE, graph=False,
          iterations=FILE, grad=False):
  c = {"model": model, "nworld": nworld, "integrator": integrator, "form": form,
       "jacobian": jacobian, "graph": graph, "iterations": iterations, "grad": grad}
  return dict(c, name=name) if name else c


def listed():
  return [
    # one simulated robot, driven interactively or by a controller: latency of one eager call
    _case("humanoid_1", "humanoid", 1, EULER),
    # the candidates of a sampling-based controller, replayed from a graph at control rate
    _case("humanoid_128_graph", "humanoid", 128, IMPLICITFAST, graph=True),
    # an odd-sized batch of environments, stepped eagerly with the model file's own integrator
    _case("humanoid_1000", "humanoid", 1000, EULER),
    # the benchmark's batch: policy training, the step captured once and replayed
    _case("humanoid_8192_graph", "humanoid", 8192, IMPLICITFAST, graph=True, iterations=BENCH),
    # the largest batch of the configurations
    _case("humanoid_32768", "humanoid", 32768, IMPLICITFAST),
    # the precision form, for runs compared against FP64 simulators
    _case("humanoid_4096_precision", "humanoid", 4096, IMPLICITFAST, form=PRECISION),
    # a small mechanism (Euler with implicit joint damping), many copies
    _case("sphere_chain_4096", "sphere_chain", 4096, EULER),
    # a robot among loose objects, uneven contact counts, both forms
    _case("spheres_4096", "humanoid_spheres", 4096, IMPLICITFAST),
    _case("spheres_1500_precision", "humanoid_spheres", 1500, IMPLICITFAST, form=PRECISION),
    # a bin of loose objects: hundreds of dofs and rows per world
    _case("bin_4096", "bin", 4096, EULER),
    # the same with the mass-matrix layout that the model gets by default, a small odd batch
    _case("bin_300_sparse", "bin", 300, EULER, jacobian=AUTO),
    # trajectory optimisation: gradients of a rollout with respect to controls and initial state
    _case("humanoid_1024_grad", "humanoid", 1024, IMPLICITFAST, grad=True),
  ]


def draw(rng):
  model = rng.choice(("humanoid", "humanoid", "humanoid", "humanoid_spheres", "bin", "sphere_chain"))
  lo, hi = MODELS[model]["worlds"]
  nworld = min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))
  integrator = EULER if model in ("bin", "sphere_chain") else rng.choice((EULER, IMPLICITFAST, IMPLICITFAST))
  c = _case(None, model, nworld, integrator, graph=rng.random() < 0.4)
  if model == "humanoid" and rng.random() < 0.3:
    c["iterations"] = BENCH
  kind = rng.random()
  if model == "bin" and kind < 0.5:
    c["jacobian"] = AUTO
  elif model != "bin" and kind < 0.2:
    c["form"] = PRECISION
  elif model == "humanoid" and kind < 0.4:
    c.update(grad=True, graph=False, iterations=FILE, integrator=IMPLICITFAST, nworld=min(nworld, 2048))
  return c


@functools.lru_cache(maxsize=None)
def _host_model(model, integrator=EULER, jacobian=DENSE, iterations=FILE, grad=False):
  mjm = mjcf.from_xml_path(os.path.join(ROOT, "tests", "golden", "models", model + ".xml"))
  mjm.opt.integrator = integrator
  if jacobian != AUTO and mjm.nv >= 60:  # below, the automatic choice is dense too
    mjm.opt.jacobian = jacobian
  if iterations == BENCH:
    mjm.opt.iterations, mjm.opt.ls_iterations = 3, 4
  if grad:  # the benchmark's differentiated rollout
    mjm.opt.iterations, mjm.opt.ls_iterations = 10, 10
  return mjm


def _state(model, mjm, n, seed):
  """Seeded (qpos, qvel, ctrl) of n worlds on the GPU."""
  g = torch.Generator(device="cuda").manual_seed(seed)

  def uniform(lo, hi, *shape):
    return torch.rand((n,) + shape, generator=g, device="cuda") * (hi - lo) + lo

  def normal(std, *shape):
    return torch.randn((n,) + shape, generator=g, device="cuda") * std

  def unit(q):
    return q / q.norm(dim=-1, keepdim=True)

  def device(x):
    return torch.as_tensor(x, dtype=torch.float32, device="cuda")

  if model.startswith("humanoid"):
    # every world in one of the humanoid's keyframes (standing, on one leg, lying), perturbed
    hum = _host_model("humanoid")
    keys = device(hum.key_qpos)
    q = keys[torch.randint(keys.shape[0], (n,), generator=g, device="cuda")]
    q = q + uniform(-0.05, 0.05, hum.nq)
    q[:, 3:7] = unit(q[:, 3:7])
    ctrl, qvel = uniform(-0.4, 0.4, mjm.nu), normal(0.01, mjm.nv)
    if model == "humanoid":
      return q, qvel, ctrl
    # k ~ U{0..16} spheres dropped next to the humanoid, the others parked far away
    nsph = (mjm.nq - hum.nq) // 7
    k = torch.randint(nsph + 1, (n, 1), generator=g, device="cuda")
    i = torch.arange(nsph, device="cuda")
    near = i < k
    s = torch.zeros((n, nsph, 7), device="cuda")
    s[:, :, 0] = torch.where(near, uniform(-0.6, 0.6, nsph), 100.0 + 2.0 * i)
    s[:, :, 1] = torch.where(near, uniform(-0.6, 0.6, nsph), 100.0)
    s[:, :, 2] = torch.where(near, uniform(0.1, 0.6, nsph), 10.0)
    s[:, :, 3] = 1.0
    return torch.cat([q, s.reshape(n, -1)], 1), qvel, ctrl
  q = device(mjm.qpos0).repeat(n, 1)
  if model == "bin":  # a seeded, overlapping packing
    b = q.view(n, mjm.nbody - 1, 7)
    b[:, :, :2] = uniform(-0.4, 0.4, mjm.nbody - 1, 2)
    b[:, :, 2] = uniform(0.03, 0.35, mjm.nbody - 1)
    b[:, :, 3:] = unit(normal(1.0, mjm.nbody - 1, 4))
    return q, normal(0.1, mjm.nv), None
  # sphere_chain: the ball just above the floor or resting in it, the chain swinging
  q[:, 2] = uniform(0.095, 0.105)
  q[:, 7:] = uniform(-0.1, 0.1, 5)
  return q, normal(0.1, mjm.nv), uniform(-1.0, 1.0, mjm.nu)


def prepare(case, seed):
  model, n, size = case["model"], case["nworld"], MODELS[case["model"]]
  mjm = _host_model(model, case["integrator"], case["jacobian"], case["iterations"], case["grad"])
  m = mjw.put_model(mjm, device="cuda")
  qpos, qvel, ctrl = _state(model, mjm, n, seed)
  if case["grad"]:
    roll = mjw.derivative.Rollout(mjm, m, n, checkpoint=CHECKPOINT, nconmax=size["nconmax"],
                                  njmax=size["njmax"])
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    u = ctrl + torch.randn((HORIZON,) + tuple(ctrl.shape), generator=g, device="cuda") * 0.05
    target = qpos[:, :3] + torch.tensor([0.05, 0.0, 0.0], device="cuda")
    return {"case": case, "roll": roll, "inputs": (qpos, qvel, u), "target": target}
  d = mjw.make_data(mjm, n, nconmax=size["nconmax"] * n, njmax=size["njmax"] * n, device="cuda")
  inputs = {"qpos": qpos, "qvel": qvel, "qacc_warmstart": torch.zeros_like(qvel)}
  if ctrl is not None:
    inputs["ctrl"] = ctrl
  state = {"case": case, "m": m, "d": d, "inputs": inputs, "out": None, "graph": None}
  if case["graph"]:
    _call(state)  # allocates the outputs, outside the capture
    torch.cuda.synchronize()
    state["graph"] = torch.cuda.CUDAGraph()
    with torch.cuda.graph(state["graph"]):
      _call(state)
  return state


def _call(state):
  state["out"] = mjw.step_io(state["m"], state["d"], 1, inputs=state["inputs"], outputs=OUTPUTS,
                             out=state["out"], fused=state["case"]["form"])
  return state["out"]


def run(state):
  if state["case"]["grad"]:
    q, v, u = (t.clone().requires_grad_(True) for t in state["inputs"])
    qT, vT = state["roll"](q, v, u)
    loss = ((qT[:, :3] - state["target"]) ** 2).sum() + 1e-3 * (u ** 2).sum()
    loss.backward()
    return {"qpos": qT.detach(), "qvel": vT.detach(), "grad_qpos": q.grad, "grad_qvel": v.grad,
            "grad_ctrl": u.grad}
  if state["graph"] is not None:
    state["graph"].replay()
    return state["out"]
  return _call(state)


def exact(case, seed):
  """No value: a pass is a whole step of the simulator (collision detection to integration), whose
  64-bit evaluation is a simulator of its own."""
  return None


def work(case):
  """Inputs read once, outputs written once; operations of the step's algorithm: smooth dynamics
  (about 600 per body), the mass matrix factored and solved tree by tree, and four Newton
  iterations of Hessian assembly and factorisation over the dofs that rows couple, products with
  the rows and line search."""
  mjm = _host_model(case["model"], case["integrator"], case["jacobian"], case["iterations"], case["grad"])
  size, n = MODELS[case["model"]], case["nworld"]
  nq, nv, nu, nb = mjm.nq, mjm.nv, mjm.nu, mjm.nbody
  tree = sum(t ** 3 / 3.0 + 2.0 * t * t for t in size["trees"])
  newton = tree + size["rows"] * (size["touched"] ** 2 + 8.0 * size["touched"] + 24.0 * 4)
  flops = n * (600.0 * nb + 2.0 * tree + 5.0 * newton)
  nbytes = 4.0 * n * (2 * nq + 4 * nv + nu + nb * (3 + 3 + 6))
  if case["grad"]:  # forward, recomputation and adjoint of every step; gradients out
    return {"bytes": 4.0 * n * (3 * nq + 3 * nv + 2 * HORIZON * nu), "flops": 3.0 * HORIZON * flops}
  return {"bytes": nbytes, "flops": flops}
