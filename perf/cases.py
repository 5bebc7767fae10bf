"""What a program that uses this solver has it do, as cases that can be timed and checked.

Each case is one call (or one short chain of calls) of the public interface on a seeded synthetic
mesh: a frame or the substep of a frame loop, the tangent refresh of a frame, a prepared step, the bare operator,
a taped differentiable substep and a checkpointed rollout gradient.  Sizes run from the 81-node
cantilever, where a substep is launches and latency, to the 64^3 Hex8 block (274,625 nodes), where the
matrix stream is twice the L2 cache; ragged grids, Tet4 and Hex8, springs, ground contact, fixed faces
and batches of uneven scenes are in between.

``exact`` restates each computation in float64 torch on the float32 inputs that the solver is given:
element forces and tangents, the matrix A = M + h^2 K + h C_s, and the block-Jacobi preconditioned
conjugate gradients with the same stopping rule.
"""

import functools
import itertools
import math

import numpy as np
import torch

from newton_solver_fem_gb300 import SolverFEM, model_from_arrays
from newton_solver_fem_gb300.adjoint import DeviceRollout, DifferentiableSolver, device_checkpointed_gradient

DEVICE = "cuda"
GRAVITY = (0.0, 0.0, -9.81)
GROUND = (300.0, 0.0, 1.0e3, 0.5)  # ke, kd, kf, mu: stable for 1 cm cells


# --------------------------------------------------------------------------------------- the cases


def listed():
    return [
        # The smallest program: a Tet4 cantilever of 81 nodes with one fixed face, a whole frame (tangent refresh,
        # then the captured graph of its substeps).
        dict(name="frame cantilever", kind="frame", element="tet", nx=8, ny=2, nz=2, cell=0.05, E=2.0e4, nu=0.45,
             rho=1000.0, fixed=True, substeps=2),
        # An interactive prop: a ragged Hex8 body of a few thousand nodes resting on the ground.
        dict(name="step hex ragged", kind="step", element="hex", nx=23, ny=17, nz=11, cell=0.01, E=5.0e5, nu=0.4,
             rho=1100.0, ground=True),
        # A detailed Tet4 body: 663,552 jittered tets with edge springs, pressed into the ground.
        dict(name="step tet springs", kind="step", element="tet", nx=48, ny=48, nz=48, cell=0.01, E=2.0e5, nu=0.45,
             rho=1000.0, jitter=0.2, springs=True, ground=True),
        # The largest single body: 64^3 Hex8 cells on the ground, matrix about twice the L2 cache.
        dict(name="step hex block", kind="step", element="hex", nx=64, ny=64, nz=64, cell=0.01, E=5.0e5, nu=0.4,
             rho=1100.0, ground=True),
        # A training or design batch: 48 independent uneven scenes, half Tet4 and half Hex8, in one handle.
        dict(name="step batch", kind="step", element="mix", nx=4, ny=32, nz=48, cell=0.05, E=0.0, nu=0.0, rho=1000.0,
             fixed=True, scenes=48, tol=1.0e-6),
        # The once-a-frame tangent refresh (element tangents, assembly, preconditioner) of a Hex8 body.
        dict(name="refresh hex", kind="refresh", element="hex", nx=48, ny=48, nz=48, cell=0.01, E=5.0e5, nu=0.4,
             rho=1100.0),
        # The same for a ragged jittered Tet4 body with springs.
        dict(name="refresh tet ragged", kind="refresh", element="tet", nx=37, ny=29, nz=22, cell=0.01, E=2.0e5,
             nu=0.45, rho=1000.0, jitter=0.2, springs=True),
        # A coupled solver's iteration: prepare the affine step, right-hand side for a load, solve, reconstruct.
        dict(name="prepared step", kind="prepared", element="hex", nx=32, ny=32, nz=32, cell=0.01, E=5.0e5, nu=0.4,
             rho=1100.0, fixed=True, tol=1.0e-4),
        # An outer Krylov method's inner products: the operator and the preconditioner on a large body.
        dict(name="operator", kind="operator", element="hex", nx=56, ny=56, nz=56, cell=0.01, E=5.0e5, nu=0.4,
             rho=1100.0, fixed=True),
        # Differentiable control of a small Tet4 beam (425 nodes): checkpointed rollout gradient with
        # respect to the initial state and per-element shear scales.
        dict(name="gradient beam", kind="gradient", element="tet", nx=4, ny=4, nz=16, cell=0.05, E=2.0e4, nu=0.45,
             rho=1000.0, fixed=True, steps=4, every=2, substeps=4),
        # One taped differentiable substep and its backward pass on a mid-size Hex8 body.
        dict(name="taped step", kind="tape", element="hex", nx=28, ny=24, nz=20, cell=0.05, E=2.0e4, nu=0.4,
             rho=1000.0, substeps=4),
        # The same rollout gradient on a larger Hex8 body, with material gradients.
        dict(name="gradient hex", kind="gradient", element="hex", nx=40, ny=36, nz=33, cell=0.05, E=2.0e4, nu=0.4,
             rho=1000.0, fixed=True, steps=2, every=2, substeps=4),
    ]


def _dims(rng, low, high):
    """Three cell counts with the node count spread over its logarithm and uneven sides."""
    side = math.exp(rng.uniform(math.log(low), math.log(high)))
    out = [max(2, min(high, round(side * rng.uniform(0.75, 1.33)))) for _ in range(3)]
    return tuple(out)


def draw(rng):
    kind = rng.choice(("step", "step", "step", "batch", "frame", "refresh", "refresh", "prepared", "operator",
                       "gradient", "tape"))
    element = rng.choice(("tet", "hex"))
    ground = rng.random() < 0.5
    E, nu = math.exp(rng.uniform(math.log(1.0e5), math.log(5.0e5))), rng.uniform(0.35, 0.45)
    if kind == "batch":
        return dict(kind="step", element="mix", nx=4, ny=rng.randint(12, 32), nz=rng.randint(1000, 9999), cell=0.05,
                    E=0.0, nu=0.0, rho=1000.0, fixed=True, scenes=rng.randint(5, 48), tol=1.0e-6)
    if kind == "frame":
        nx, ny, nz = _dims(rng, 2, 12)
        return dict(kind=kind, element=element, nx=nx, ny=ny, nz=nz, cell=0.05, E=0.1 * E, nu=nu, rho=1000.0, fixed=True,
                    substeps=2)
    if kind in ("gradient", "tape"):
        small = rng.random() < 0.5
        nx, ny, nz = _dims(rng, 3, 8) if small else _dims(rng, 8, 30)
        c = dict(kind=kind, element=element, nx=nx, ny=ny, nz=nz, cell=0.05, E=0.1 * E, nu=nu, rho=1000.0, substeps=4)
        if kind == "gradient":
            every = rng.randint(1, 2)
            c.update(fixed=True, every=every, steps=every * rng.randint(1, 2))
        return c
    top = 56 if element == "hex" else 46
    nx, ny, nz = _dims(rng, 3, top)
    c = dict(kind=kind, element=element, nx=nx, ny=ny, nz=nz, cell=0.01, E=E, nu=nu, rho=1000.0)
    if element == "tet" and rng.random() < 0.7:
        c["jitter"] = 0.2
        c["springs"] = rng.random() < 0.6
    if kind == "step":
        c["ground" if ground else "fixed"] = True
    elif kind in ("prepared", "operator"):
        c["fixed"] = True
    if kind == "prepared":
        c["tol"] = 1.0e-4
    return c


# --------------------------------------------------------------------------------------- the meshes

_SIGNS = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]],
                  dtype=np.float64)


def _shape(points):
    factors = 1.0 + points[:, None, :] * _SIGNS[None]
    values = np.prod(factors, axis=2) / 8.0
    deriv = np.empty((len(points), 8, 3))
    for d in range(3):
        a, b = (k for k in range(3) if k != d)
        deriv[:, :, d] = _SIGNS[None, :, d] * factors[:, :, a] * factors[:, :, b] / 8.0
    return values, deriv


_POINTS = _SIGNS / math.sqrt(3.0)
_VALUES, _DERIV = _shape(_POINTS)  # [8 points, 8 nodes], [8 points, 8 nodes, 3]


def _grid(nx, ny, nz, cell):
    k, j, i = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
    return np.stack([i.ravel(), j.ravel(), k.ravel()], 1), np.stack([i.ravel(), j.ravel(), k.ravel()], 1) * float(cell)


def _corners(nx, ny, nz):
    k, j, i = (a.ravel() for a in np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij"))
    return lambda b: (i + b[0]) + (nx + 1) * ((j + b[1]) + (ny + 1) * (k + b[2]))


def _hexes(nx, ny, nz):
    at = _corners(nx, ny, nz)
    return np.stack([at(((s + 1) // 2).astype(int)) for s in _SIGNS], 1).astype(np.int32)


def _tets(nx, ny, nz):
    """Six tets per cell along the paths from corner (0,0,0) to (1,1,1), positively oriented."""
    at = _corners(nx, ny, nz)
    out = []
    for order in itertools.permutations(range(3)):
        p = [np.zeros(3, int)]
        for axis in order:
            p.append(p[-1] + np.eye(3, dtype=int)[axis])
        if np.linalg.det(np.array([p[1], p[2], p[3]], float)) < 0:
            p[2], p[3] = p[3], p[2]
        out.append(np.stack([at(b) for b in p], 1))
    return np.stack(out, 1).reshape(-1, 4).astype(np.int32)


def _one_mesh(element, nx, ny, nz, cell, E, nu, rho, jitter, rng):
    ijk, x = _grid(nx, ny, nz, cell)
    if jitter:
        inside = np.all((ijk > 0) & (ijk < (nx, ny, nz)), axis=1)
        x[inside] += rng.uniform(-jitter * cell, jitter * cell, (int(inside.sum()), 3))
    mats = (E / (2.0 * (1.0 + nu)), E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)), 0.0)
    if element == "tet":
        el = _tets(nx, ny, nz)
        share = np.repeat(rho * np.linalg.det(x[el[:, 1:]] - x[el[:, :1]]) / 24.0, 4)
    else:
        el = _hexes(nx, ny, nz)
        if jitter:
            det = np.linalg.det(np.einsum("hai,gaj->hgij", x[el], _DERIV))
        else:
            det = np.full((len(el), 8), (cell / 2.0) ** 3)
        share = (rho * det @ _VALUES).ravel()
    mass = np.bincount(el.ravel(), weights=share, minlength=len(x))
    fixed = np.nonzero(ijk[:, 0] == 0)[0]
    return x, el, np.tile(np.array(mats, np.float32), (len(el), 1)), mass, fixed


@functools.lru_cache(maxsize=2)
def _mesh(element, nx, ny, nz, cell, E, nu, rho, jitter, springs, scenes):
    """Host arrays of a case's body (or batch of bodies), the same for every seed."""
    rng = np.random.default_rng(5 if scenes == 1 else 1000 * scenes + nz)
    xs, masses, fixed, offsets, start = [], [], [], [0], 0
    el = {"tet": [], "hex": []}
    mats = {"tet": [], "hex": []}
    for s in range(scenes):
        kind, dims, e, p = element, (nx, ny, nz), E, nu
        if element == "mix":
            kind, dims = ("tet", "hex")[s % 2], tuple(int(v) for v in rng.integers(nx, ny + 1, 3))
            e, p = math.exp(rng.uniform(math.log(1.0e4), math.log(1.0e6))), rng.uniform(0.3, 0.48)
        x, c, m, mass, f = _one_mesh(kind, *dims, cell, e, p, rho, jitter, rng)
        el[kind].append(c + start)
        mats[kind].append(m)
        xs.append(x)
        masses.append(mass)
        fixed.append(f + start)
        start += len(x)
        offsets.append(start)
    out = dict(x=np.concatenate(xs), mass=np.concatenate(masses), fixed=np.concatenate(fixed).astype(np.int32),
               offsets=np.array(offsets, np.int64) if scenes > 1 else None)
    for k, n in (("tet", 4), ("hex", 8)):
        out[k] = np.concatenate(el[k]) if el[k] else np.zeros((0, n), np.int32)
        out[k + "_mats"] = np.concatenate(mats[k]) if mats[k] else np.zeros((0, 3), np.float32)
    out["springs"] = np.zeros((0, 2), np.int32)
    if springs and len(out["tet"]):
        t = out["tet"].astype(np.int64)
        pairs = np.concatenate([np.sort(t[:, list(p)], 1) for p in itertools.combinations(range(4), 2)])
        keys = np.unique(pairs[:, 0] * len(out["x"]) + pairs[:, 1])
        out["springs"] = np.stack([keys // len(out["x"]), keys % len(out["x"])], 1).astype(np.int32)
    return out


def _body(case):
    return _mesh(case["element"], case["nx"], case["ny"], case["nz"], case["cell"], case["E"], case["nu"], case["rho"],
                 case.get("jitter", 0.0), bool(case.get("springs")), case.get("scenes", 1))


def _dt(case):
    return 1.0 / (60.0 * case.get("substeps", 10))


def _inputs(case, seed):
    """The seeded state of a body in motion: a smooth deformation of several percent strain and a smooth velocity
    with some noise on both, the last substep's increment, a load, shear scales and output gradients."""
    body = _body(case)
    rng = np.random.default_rng(seed)
    x, cell = body["x"], case["cell"]
    n = len(x)
    q, v = x.copy(), rng.normal(0.0, 0.05, x.shape)
    for _ in range(3):
        wave = rng.uniform(-1.0, 1.0, 3) * (2.0 * math.pi / (12.0 * cell))
        q += 0.1 * cell * np.sin(x @ wave + rng.uniform(0.0, 6.28))[:, None] * rng.uniform(-1.0, 1.0, 3)
        v += 20.0 * cell * np.sin(x @ wave + rng.uniform(0.0, 6.28))[:, None] * rng.uniform(-1.0, 1.0, 3)
    q += rng.normal(0.0, 0.01 * cell, x.shape)
    dv = rng.normal(0.0, 2.0e-3, x.shape) + np.array(GRAVITY) * _dt(case)
    if case.get("ground"):
        q[:, 2] -= 0.02 * cell  # the bottom layer presses into the plane z = 0
    load = rng.normal(0.0, 1.0, x.shape) * body["mass"][:, None] * 5.0
    if case.get("fixed"):
        held = body["fixed"]
        q[held], v[held], dv[held] = x[held], 0.0, 0.0
    f32 = lambda a: np.ascontiguousarray(a, dtype=np.float32)  # noqa: E731
    return {"q": f32(q), "v": f32(v), "dv": f32(dv), "load": f32(load), "scale": f32(rng.uniform(0.8, 1.2, len(body["tet"]))),
            "gq": f32(rng.normal(0.0, 1.0, (n, 3)) / cell), "gv": f32(rng.normal(0.0, 1.0, (n, 3)))}


# --------------------------------------------------------------------------------------- the framework


def prepare(case, seed):
    body, inp = _body(case), _inputs(case, seed)
    kind = case["kind"]
    ns = len(body["springs"])
    model = model_from_arrays(
        body["x"], body["mass"], tets=body["tet"] if len(body["tet"]) else None, tet_materials=body["tet_mats"],
        hexes=body["hex"] if len(body["hex"]) else None, hex_materials=body["hex_mats"], springs=body["springs"],
        spring_ke=np.full(ns, 1.0e3, np.float32), spring_kd=np.full(ns, 0.1, np.float32), radius=0.0, gravity=GRAVITY,
        scene_offsets=body["offsets"], device=DEVICE)
    ke, kd, kf, mu = GROUND
    tape = kind == "tape"
    solver = SolverFEM(
        model, dt=_dt(case), solver_type="cg", preconditioner_type="block_diag",
        linear_solver_maxiter=30 if kind in ("tape", "gradient") else 50, linear_solver_tolerance=case.get("tol", 1.0e-2),
        ground_plane=(0.0, 0.0, 1.0, 0.0) if case.get("ground") else None, ground_ke=ke, ground_kd=kd, ground_kf=kf,
        ground_mu=mu, self_contact_ke=0.0, fixed_particle_indices=body["fixed"] if case.get("fixed") else None,
        differentiable=tape, defer_differentiation_checks=tape)
    dev = {k: torch.as_tensor(a, device=DEVICE) for k, a in inp.items()}
    a, b = model.state(), model.state()
    a.particle_q.copy_(dev["q"])
    a.particle_qd.copy_(dev["v"])
    state = dict(case=case, solver=solver, model=model, a=a, b=b, **dev)
    if kind in ("step", "prepared", "operator"):
        solver.refresh_tangent(a.particle_q)  # the frame's tangent, taken where the frame began
    if kind == "operator":
        state["step"] = solver.prepare_step(a, None, None, _dt(case))
        state["out_a"], state["out_b"] = torch.empty_like(dev["gv"]), torch.empty_like(dev["gv"])
    if kind == "gradient":
        state["diff"] = DifferentiableSolver(solver, tolerance=1.0e-8, maxiter=30)
        state["rollout"] = DeviceRollout(state["diff"], case["steps"], case["every"])
        state["target"] = dev["q"] - 0.5 * case["cell"]
    if kind == "frame":  # the substep loop as a graph, captured once after a warm-up
        state["graph"] = graph = torch.cuda.CUDAGraph()
        solver.refresh_tangent(a.particle_q)
        solver.step(a, b, None, None, solver.dt)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            for i in range(case["substeps"]):
                solver.step(*((a, b) if i % 2 == 0 else (b, a)), None, None, solver.dt)
    if tape:
        solver.prepare_differentiation()
    return state


def _run_step(s):
    solver, a, b = s["solver"], s["a"], s["b"]
    solver.velocity_increment.copy_(s["dv"])  # the warm start that the substep before this one left
    solver.step(a, b, None, None, solver.dt)
    return [b.particle_q, b.particle_qd, solver.velocity_increment, a.particle_f]


def _run_frame(s):
    solver, a = s["solver"], s["a"]
    a.particle_q.copy_(s["q"])
    a.particle_qd.copy_(s["v"])
    solver.velocity_increment.copy_(s["dv"])
    solver.refresh_tangent(a.particle_q)
    s["graph"].replay()
    return [a.particle_q, a.particle_qd]


def _run_refresh(s):
    s["solver"].refresh_tangent(s["a"].particle_q)
    A = s["solver"].A_bsr  # the matrix as a program takes it, canonical block-row order
    return [A.offsets, A.columns, A.values]


def _run_prepared(s):
    solver = s["solver"]
    solver.velocity_increment.copy_(s["dv"])
    step = solver.prepare_step(s["a"], None, None, solver.dt)
    rhs = step.rhs(s["load"])
    dv = step.solve(rhs, tolerance=s["case"]["tol"])
    step.reconstruct(dv, s["b"])
    return [step.base_rhs, rhs, step.diagonal_blocks, dv, s["b"].particle_q, s["b"].particle_qd]


def _run_operator(s):
    s["step"].apply_operator(s["gv"], s["out_a"])
    s["step"].apply_preconditioner(s["gq"], s["out_b"])
    return [s["out_a"], s["out_b"]]


def _run_gradient(s):
    target = s["target"]
    loss, grads = device_checkpointed_gradient(
        s["diff"], s["q"], s["v"], s["case"]["steps"], s["case"]["every"],
        lambda q, v: 0.5 * ((q - target) ** 2).sum() + 1.0e-4 * (v ** 2).sum(),
        mu_scale=s["scale"] if len(s["scale"]) else None, materials=len(s["scale"]) == 0, rollout=s["rollout"])
    return {"loss": loss, **grads}


def _run_tape(s):
    solver, model = s["solver"], s["model"]
    a, b = model.state(), model.state()
    a.particle_q = s["q"].detach().requires_grad_(True)
    a.particle_qd = s["v"].detach().requires_grad_(True)
    load = s["load"].detach().requires_grad_(True)
    solver.step(a, b, None, None, solver.dt, external_forces=load)
    grads = torch.autograd.grad((b.particle_q, b.particle_qd), (a.particle_q, a.particle_qd, load), (s["gq"], s["gv"]))
    return [b.particle_q, b.particle_qd, *grads]


_RUN = {"step": _run_step, "frame": _run_frame, "refresh": _run_refresh, "prepared": _run_prepared, "operator": _run_operator,
        "gradient": _run_gradient, "tape": _run_tape}


def run(state):
    return _RUN[state["case"]["kind"]](state)


# --------------------------------------------------------------------------------------- bytes and operations


def _counts(case):
    """Nodes, tets, hexes, springs and matrix blocks; a grid's blocks from its neighbour stencil."""
    def one(kind, nx, ny, nz):
        n = (nx + 1) * (ny + 1) * (nz + 1)
        if kind == "hex":
            return n, 0, nx * ny * nz, (3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)
        pairs = 0
        for d in ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1)):
            pairs += (nx + 1 - d[0]) * (ny + 1 - d[1]) * (nz + 1 - d[2])
        return n, 6 * nx * ny * nz, 0, n + 2 * pairs

    if case["element"] != "mix":
        n, t, h, z = one(case["element"], case["nx"], case["ny"], case["nz"])
        return n, t, h, (z - n) // 2 if case.get("springs") else 0, z
    rng = np.random.default_rng(1000 * case["scenes"] + case["nz"])
    total = np.zeros(4, np.int64)
    for s in range(case["scenes"]):
        dims = [int(v) for v in rng.integers(case["nx"], case["ny"] + 1, 3)]
        rng.uniform(0.0, 1.0), rng.uniform(0.0, 1.0)
        total += one(("tet", "hex")[s % 2], *dims)
    n, t, h, z = (int(v) for v in total)
    return n, t, h, 0, z


def work(case):
    """Every input once and every output once; the matrix is an input of a solve (36 B a block and its column)."""
    n, t, h, s, z = _counts(case)
    matrix, elements, state = 40 * z, 64 * t + 364 * h + 20 * s, 24 * n
    element_flops = 400 * t + 5000 * h + 40 * s
    solve = 18 * z + 80 * n  # one conjugate-gradient iteration
    its = {1.0e-2: 12, 1.0e-4: 22, 1.0e-6: 34}.get(case.get("tol", 1.0e-2), 30)
    kind = case["kind"]
    if kind == "step":
        return {"bytes": matrix + elements + 2 * state + 36 * n + 24 * n, "flops": element_flops + (its + 2) * solve}
    if kind == "frame":
        return {"bytes": matrix + elements + 2 * state + 36 * n + 12 * n,
                "flops": case["substeps"] * (element_flops + (its + 2) * solve) + 1200 * t + 20000 * h}
    if kind == "refresh":
        return {"bytes": elements + 12 * n + 40 * z + 36 * n, "flops": 1200 * t + 20000 * h}
    if kind == "prepared":
        return {"bytes": matrix + elements + 2 * state + 12 * n + 36 * n + 36 * n + 12 * n + 36 * n,
                "flops": element_flops + (its + 2) * solve}
    if kind == "operator":
        return {"bytes": matrix + 24 * n + 36 * n + 24 * n, "flops": 18 * z + 18 * n}
    if kind == "tape":
        return {"bytes": matrix + elements + 3 * state + 36 * n + 2 * state, "flops": 3 * element_flops + 62 * solve}
    k = case["steps"]
    return {"bytes": matrix + elements + 36 * n + 4 * state + 12 * max(t, h) + 2 * k * state,
            "flops": k * (4 * element_flops + 93 * solve)}


# --------------------------------------------------------------------------------------- the same in 64 bits


class _Exact:
    """Forces, tangents, matrix products and conjugate gradients in float64, on the solver's float32 inputs."""

    def __init__(self, case):
        body = _body(case)
        self.case = case
        up = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=DEVICE)  # noqa: E731
        r32 = lambda a: np.asarray(a, np.float32)  # noqa: E731
        idx = lambda a: torch.as_tensor(np.asarray(a, np.int64), device=DEVICE)  # noqa: E731
        x = body["x"]
        self.n = len(x)
        self.rest, self.mass = up(r32(x)), up(r32(body["mass"]))
        self.h = float(np.float32(_dt(case)))
        self.g = up(r32(GRAVITY))
        self.fixed = torch.zeros(self.n, dtype=torch.bool, device=DEVICE)
        if case.get("fixed"):
            self.fixed[idx(body["fixed"])] = True
        off = body["offsets"] if body["offsets"] is not None else np.array([0, self.n])
        self.scenes = len(off) - 1
        self.scene = idx(np.repeat(np.arange(self.scenes), np.diff(off)))
        self.tet, self.hex, self.spr = idx(body["tet"]), idx(body["hex"]), idx(body["springs"])
        self.tm, self.hm = up(body["tet_mats"]), up(body["hex_mats"])
        if len(self.tet):
            e = (x[body["tet"][:, 1:]] - x[body["tet"][:, :1]]).transpose(0, 2, 1)
            self.Dm = up(r32(np.linalg.inv(e)))
        if len(self.hex):
            J = np.einsum("hai,gaj->hgij", x[body["hex"]], _DERIV)
            self.iJ, self.w = up(r32(np.linalg.inv(J))), up(r32(np.abs(np.linalg.det(J))))
            self.dN = torch.einsum("gaj,hgji->hgai", up(r32(_DERIV)), self.iJ)
        if len(self.spr):
            p = x[body["springs"]]
            self.rest_len = up(r32(np.linalg.norm(p[:, 0] - p[:, 1], axis=1)))
        self.ke, self.kd = float(np.float32(1.0e3)), float(np.float32(0.1))
        self.ground = [float(np.float32(v)) for v in GROUND]

    # -- forces at (q, v); mu_scale multiplies the shear modulus of each tet
    def forces(self, q, v, mu_scale=None, hm=None):
        f = torch.zeros_like(q)
        if len(self.tet):
            mu = self.tm[:, 0] if mu_scale is None else self.tm[:, 0] * mu_scale
            lam, kd = self.tm[:, 1], self.tm[:, 2]
            V = 1.0 / (6.0 * torch.linalg.det(self.Dm))
            e = q[self.tet[:, 1:]] - q[self.tet[:, :1]]
            ve = v[self.tet[:, 1:]] - v[self.tet[:, :1]]
            F = e.transpose(1, 2) @ self.Dm
            dF = ve.transpose(1, 2) @ self.Dm
            Ic = (F * F).sum((1, 2))
            P = F * (mu * V * (1.0 - 1.0 / (Ic + 1.0)))[:, None, None] + dF * (kd * V)[:, None, None]
            d = torch.stack([torch.linalg.cross(e[:, 1], e[:, 2]), torch.linalg.cross(e[:, 2], e[:, 0]),
                             torch.linalg.cross(e[:, 0], e[:, 1])], 1) / (6.0 * V)[:, None, None]
            J = torch.linalg.det(F).clamp(min=0.01)
            press = (J - (1.0 + 0.75 * mu / lam)) * lam * V + (d * ve).sum((1, 2)) * kd * V
            fa = (P @ self.Dm.transpose(1, 2)).transpose(1, 2) + d * press[:, None, None]
            f = f.index_add(0, self.tet[:, 1:].reshape(-1), -fa.reshape(-1, 3))
            f = f.index_add(0, self.tet[:, 0], fa.sum(1))
        if len(self.hex):
            m = self.hm if hm is None else hm
            mu, lam, kd = (m[:, k, None, None, None] for k in range(3))
            F = torch.einsum("hai,hgaj->hgij", q[self.hex], self.dN)
            dF = torch.einsum("hai,hgaj->hgij", v[self.hex], self.dN)
            Ic = (F * F).sum((2, 3), keepdim=True)
            J = torch.linalg.det(F).clamp(min=0.01)[..., None, None]
            P = F * (mu * (1.0 - 1.0 / (Ic + 1.0))) + dF * kd + self.cof(F) * (lam * (J - (1.0 + 0.75 * mu / lam)))
            fa = -torch.einsum("hgij,hgaj,hg->hai", P, self.dN, self.w)
            f = f.index_add(0, self.hex.reshape(-1), fa.reshape(-1, 3))
        if len(self.spr):
            a, b = self.spr[:, 0], self.spr[:, 1]
            xij, vij = q[a] - q[b], v[a] - v[b]
            L = xij.norm(dim=1)
            u = xij / L[:, None]
            fs = u * (self.ke * (L - self.rest_len) + self.kd * (u * vij).sum(1))[:, None]
            f = f.index_add(0, a, -fs).index_add(0, b, fs)
        if self.case.get("ground"):
            ke, kd, kf, mu = self.ground
            c = q[:, 2].clamp(max=0.0)
            vn = v[:, 2]
            fn = c * ke + vn.clamp(max=0.0) * kd
            vt = v * torch.tensor([1.0, 1.0, 0.0], device=q.device, dtype=q.dtype)
            vs = vt.norm(dim=1)
            fe = torch.minimum(fn.abs(), self.mass * self.g.norm())
            ft = torch.minimum(vs * kf, mu * fe)
            hit = torch.zeros_like(f)
            hit[:, 2] = -fn
            hit = hit - vt / vs.clamp(min=1e-300)[:, None] * ft[:, None]
            f = f + torch.where((c < 0.0)[:, None], hit, torch.zeros_like(hit))
        return f + self.mass[:, None] * self.g

    @staticmethod
    def cof(F):
        c = [F[..., :, k] for k in range(3)]
        return torch.stack([torch.linalg.cross(c[1], c[2]), torch.linalg.cross(c[2], c[0]),
                            torch.linalg.cross(c[0], c[1])], -1)

    # -- the matrix at q: element matrices and the constant part
    def assemble(self, q):
        h2 = self.h * self.h
        self.Kt = self.Kh = None
        eye = torch.eye(3, dtype=torch.float64, device=DEVICE)
        if len(self.tet):
            mu, lam = self.tm[:, 0], self.tm[:, 1]
            V = 1.0 / (6.0 * torch.linalg.det(self.Dm))
            e = q[self.tet[:, 1:]] - q[self.tet[:, :1]]
            F = e.transpose(1, 2) @ self.Dm
            Ic1 = (F * F).sum((1, 2)) + 1.0
            d = torch.stack([torch.linalg.cross(e[:, 1], e[:, 2]), torch.linalg.cross(e[:, 2], e[:, 0]),
                             torch.linalg.cross(e[:, 0], e[:, 1])], 1) / (6.0 * V)[:, None, None]
            dJ = torch.cat([-d.sum(1, keepdim=True), d], 1)
            dm = torch.cat([-self.Dm.sum(1, keepdim=True), self.Dm], 1)
            Fd = torch.einsum("tij,taj->tai", F, dm)
            K = torch.einsum("tai,tbj->taibj", Fd, Fd) * (2.0 * mu * V / Ic1 ** 2)[:, None, None, None, None]
            K += torch.einsum("tai,tbj->taibj", dJ, dJ) * (lam * V)[:, None, None, None, None]
            dd = torch.einsum("taj,tbj->tab", dm, dm) * (mu * V * (1.0 - 1.0 / Ic1))[:, None, None]
            K += dd[:, :, None, :, None] * eye[None, None, :, None, :]
            self.Kt = (K * h2).reshape(-1, 12, 12)
        if len(self.hex):
            F = torch.einsum("hai,hgaj->hgij", q[self.hex], self.dN)
            Ic1 = (F * F).sum((2, 3)) + 1.0
            c1 = self.hm[:, None, 0] * (1.0 - 1.0 / Ic1) * self.w
            c2 = 2.0 * self.hm[:, None, 0] / Ic1 ** 2 * self.w
            c3 = self.hm[:, None, 1] * self.w
            fd = torch.einsum("hgij,hgaj->hgai", F, self.dN).reshape(-1, 8, 24)
            cd = torch.einsum("hgij,hgaj->hgai", self.cof(F), self.dN).reshape(-1, 8, 24)
            K = torch.baddbmm((fd * c2[..., None]).transpose(1, 2) @ fd, (cd * c3[..., None]).transpose(1, 2), cd)
            dd = torch.einsum("hgaj,hgbj,hg->hab", self.dN, self.dN, c1)
            K = K.reshape(-1, 8, 3, 8, 3)
            for k in range(3):
                K[:, :, k, :, k] += dd
            self.Kh = (K * h2).reshape(-1, 24, 24)
        self.cs = self.h * self.kd + h2 * self.ke
        diag = self.mass[:, None, None] * eye
        for el, K in ((self.tet, self.Kt), (self.hex, self.Kh)):
            if K is not None:
                w = el.shape[1]
                blocks = torch.stack([K[:, 3 * a:3 * a + 3, 3 * a:3 * a + 3] for a in range(w)], 1)
                diag = diag.index_add(0, el.reshape(-1), blocks.reshape(-1, 3, 3))
        if len(self.spr):
            diag = diag.index_add(0, self.spr.reshape(-1), (self.cs * eye).expand(2 * len(self.spr), 3, 3))
        self.diag = diag
        self.minv = torch.linalg.inv(diag)
        return self

    def stiff(self, p):
        """(A - M) p."""
        y = torch.zeros_like(p)
        for el, K in ((self.tet, self.Kt), (self.hex, self.Kh)):
            if K is not None:
                ye = torch.bmm(K, p[el].reshape(len(el), -1, 1))
                y = y.index_add(0, el.reshape(-1), ye.reshape(-1, 3))
        if len(self.spr):
            a, b = self.spr[:, 0], self.spr[:, 1]
            d = (p[a] - p[b]) * self.cs
            y = y.index_add(0, a, d).index_add(0, b, -d)
        return y

    def product(self, p):
        """(P A P + I - P) p."""
        keep = ~self.fixed[:, None]
        y = self.stiff(p * keep) + self.mass[:, None] * p * keep
        return torch.where(keep, y, p)

    def bsr(self):
        """Offsets, columns and values in canonical order (rows, then columns, ascending)."""
        rows, cols, vals = [], [], []
        ids = torch.arange(self.n, device=DEVICE)
        eye = torch.eye(3, dtype=torch.float64, device=DEVICE)
        rows.append(ids)
        cols.append(ids)
        vals.append(self.mass[:, None, None] * eye)
        for el, K in ((self.tet, self.Kt), (self.hex, self.Kh)):
            if K is not None:
                w = el.shape[1]
                rows.append(el[:, :, None].expand(-1, w, w).reshape(-1))
                cols.append(el[:, None, :].expand(-1, w, w).reshape(-1))
                vals.append(K.reshape(-1, w, 3, w, 3).transpose(2, 3).reshape(-1, 3, 3))
        if len(self.spr):
            a, b = self.spr[:, 0], self.spr[:, 1]
            block = (self.cs * eye).expand(len(a), 3, 3)
            for r, c, s in ((a, a, 1.0), (b, b, 1.0), (a, b, -1.0), (b, a, -1.0)):
                rows.append(r)
                cols.append(c)
                vals.append(s * block)
        key, slot = torch.unique(torch.cat(rows) * self.n + torch.cat(cols), return_inverse=True)
        out = torch.zeros((len(key), 3, 3), dtype=torch.float64, device=DEVICE).index_add(0, slot, torch.cat(vals))
        offsets = torch.zeros(self.n + 1, dtype=torch.int64, device=DEVICE)
        offsets[1:] = torch.cumsum(torch.bincount(key // self.n, minlength=self.n), 0)
        return offsets.to(torch.int32), (key % self.n).to(torch.int32), out

    def rhs(self, q, v, load=None, mu_scale=None):
        f = self.forces(q, v, mu_scale)
        r = self.h * (f if load is None else f + load) - self.stiff(v)
        if len(self.spr):
            a, b = self.spr[:, 0], self.spr[:, 1]
            c = (v[a] - v[b]) * (self.h * self.kd)
            r = r.index_add(0, a, c).index_add(0, b, -c)
        return torch.where(self.fixed[:, None], torch.zeros_like(r), r)

    def solve(self, b, x, tol, most):
        """Conjugate gradients, each scene with its own scalars, until ||r||^2 <= tol^2 ||b||^2."""
        per = lambda u, w: torch.zeros(self.scenes, dtype=torch.float64, device=DEVICE).index_add(  # noqa: E731
            0, self.scene, (u * w).sum(1))
        tol = float(np.float32(tol))
        r = b - self.product(x)
        z = torch.einsum("nij,nj->ni", self.minv, r)
        stop = tol * tol * per(b, b)
        rz, p = per(r, z), z
        active = per(r, r) > stop
        for _ in range(most):
            if not bool(active.any()):
                break
            y = self.product(p)
            alpha = torch.where(active, rz / per(p, y), torch.zeros_like(rz))[self.scene][:, None]
            x, r = x + alpha * p, r - alpha * y
            z = torch.einsum("nij,nj->ni", self.minv, r)
            new = per(r, z)
            beta = torch.where(active, new / rz, torch.zeros_like(new))
            rz = torch.where(active, new, rz)
            p = z + beta[self.scene][:, None] * p
            active = active & (per(r, r) > stop)
        return x

    def advance(self, q, v, dv):
        v1 = v + dv
        q1 = q + self.h * v1
        held = self.fixed[:, None]
        return torch.where(held, self.rest, q1), torch.where(held, torch.zeros_like(v1), v1)


def exact(case, seed):
    ex = _Exact(case)
    inp = {k: torch.as_tensor(a.astype(np.float64), device=DEVICE) for k, a in _inputs(case, seed).items()}
    q, v, kind = inp["q"], inp["v"], case["kind"]
    tol = case.get("tol", 1.0e-2)
    if kind == "refresh":
        return list(ex.assemble(q).bsr())
    if kind == "operator":
        ex.assemble(q)
        return [ex.product(inp["gv"]), torch.einsum("nij,nj->ni", ex.minv, inp["gq"])]
    if kind == "step":
        b = ex.assemble(q).rhs(q, v)
        dv = ex.solve(b, inp["dv"], tol, 50)
        q1, v1 = ex.advance(q, v, dv)
        return [q1, v1, dv, b]
    if kind == "frame":
        ex.assemble(q)
        dv = inp["dv"]
        for _ in range(case["substeps"]):
            dv = ex.solve(ex.rhs(q, v), dv, tol, 50)
            q, v = ex.advance(q, v, dv)
        return [q, v]
    if kind == "prepared":
        ex.assemble(q)
        base, b = ex.rhs(q, v), ex.rhs(q, v, inp["load"])
        dv = ex.solve(b, inp["dv"], tol, 50)
        q1, v1 = ex.advance(q, v, dv)
        eye = torch.eye(3, dtype=torch.float64, device=DEVICE)
        return [base, b, torch.where(ex.fixed[:, None, None], eye, ex.diag), dv, q1, v1]
    ex.assemble(ex.rest)  # the differentiable contract: the matrix of the rest state, held fixed
    scale = inp["scale"] if kind == "gradient" and len(inp["scale"]) else None
    load = inp["load"] if kind == "tape" else None
    hm = ex.hm.clone()
    zero = torch.zeros_like(q)

    def forward(q, v):
        return ex.advance(q, v, ex.solve(ex.rhs(q, v, load, scale), zero, 1.0e-8, 30))

    def backward(q, v, qb, vb):
        held = ex.fixed[:, None]
        qb, vb = torch.where(held, zero, qb), torch.where(held, zero, vb)
        vt = vb + ex.h * qb
        rb = ex.solve(vt, zero, 1.0e-8, 30)
        with torch.enable_grad():
            ins = [q.clone().requires_grad_(True), v.clone().requires_grad_(True)]
            extra = [t.clone().requires_grad_(True) for t in ([scale] if scale is not None else [hm])]
            f = ex.forces(*ins, *(extra if scale is not None else [None, extra[0]]))
            got = torch.autograd.grad(f, ins + extra, ex.h * rb, allow_unused=True)
        got = [torch.zeros_like(t) if g is None else g for g, t in zip(got, ins + extra)]
        q0, v0 = qb + got[0], vt - ex.stiff(rb) + got[1]
        if len(ex.spr):
            a, b = ex.spr[:, 0], ex.spr[:, 1]
            c = (rb[a] - rb[b]) * (ex.h * ex.kd)
            v0 = v0.index_add(0, a, c).index_add(0, b, -c)
        return torch.where(held, zero, q0), torch.where(held, zero, v0), got[2], ex.h * rb

    if kind == "tape":
        q1, v1 = forward(q, v)
        gq, gv, _, gl = backward(q, v, inp["gq"], inp["gv"])
        return [q1, v1, gq, gv, gl]
    states = [(q, v)]
    for _ in range(case["steps"]):
        states.append(forward(*states[-1]))
    target = (torch.as_tensor(_inputs(case, seed)["q"], device=DEVICE) - 0.5 * case["cell"]).double()
    qf, vf = states[-1]
    loss = 0.5 * ((qf - target) ** 2).sum() + 1.0e-4 * (vf ** 2).sum()
    qb, vb, controls = qf - target, 2.0e-4 * vf, 0.0
    for q, v in reversed(states[:-1]):
        qb, vb, c, _ = backward(q, v, qb, vb)
        controls = controls + c
    return {"loss": loss, "q0": qb, "v0": vb, ("mu_scale" if scale is not None else "hex_materials"): controls}
