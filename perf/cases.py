"""The framework's work in use, as cases to measure.

A user of this framework evaluates element forces on tetrahedral meshes, solves linear static
problems (one mesh, or a batch of meshes), advances implicit steps with the first-order
solvers (one body, or a batch of sequences), and trains the warm-start network.  Each case is
one such call sequence through the public classes.  Meshes are straight-sided tetrahedra, as
TetGen and the structured mesher give them: beams whose inner corner nodes are moved at
random by up to a tenth of a cell, TET10 mid-edge nodes at the edge midpoints.  Solves run to
the solver's default tolerance of 1e-10, where that takes up to some tenths of a second; the
large ones run the budget of iterations that a user gives as max_iter.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import tlfea_b200 as T
from tlfea_b200 import mesh as M

RHO = 1000.0
DEV = "cuda"


# ------------------------------------------------------------------------------- the cases


def listed():
    return [
        # Internal force of a fine beam after an explicit integrator has moved its nodes on the
        # device: the mesh of the large single-mesh benchmark, 480,000 elements.
        dict(name="force_t10_fp64_large", kind="force", nx=200, ny=20, nz=20, order=10, precision="fp64", damped=False),
        # The same with FP32 element arithmetic on an ordinary mesh (the time-stepping beam).
        dict(name="force_t10_fp32", kind="force", nx=100, ny=10, nz=10, order=10, precision="fp32", damped=False),
        # A small linear-tetrahedron part with Kelvin-Voigt damping: one launch-bound call.
        dict(name="force_t4_damped_small", kind="force", nx=31, ny=7, nz=5, order=4, precision="fp64", damped=True),
        # The 240-element cantilever of the reference's examples, solved to the default tolerance.
        dict(name="static_small", kind="static", nx=10, ny=2, nz=2, order=10, tol=1e-10, max_iter=10000),
        # An ordinary single linear static solve (the learned warm start's mesh).
        dict(name="static_mid", kind="static", nx=40, ny=8, nz=8, order=10, tol=1e-10, max_iter=20000),
        # A large one: 2.0 million DOF.
        dict(name="static_large", kind="static", nx=200, ny=20, nz=20, order=10, tol=1e-10, max_iter=100),
        # Two implicit steps with a time-varying load by the reference's Nesterov solver.
        dict(name="nesterov_mid", kind="step", nx=40, ny=8, nz=8, order=10, solver="nesterov", precision="fp64",
             steps=2, max_outer=2, max_inner=60),
        # One implicit step of a large body with FP32 element forces.
        dict(name="nesterov_large_fp32", kind="step", nx=120, ny=18, nz=18, order=10, solver="nesterov",
             precision="fp32", steps=1, max_outer=1, max_inner=60),
        # A design study: many uneven cantilevers of different size and material in one batch.
        dict(name="batch_uneven", kind="batch", instances=48, nx_max=48, ny_max=6, layout=1, shared=False,
             tol=1e-10, max_iter=20000),
        # Many load cases and materials on one mesh, from a predicted start.
        dict(name="batch_shared_warm", kind="batch", instances=64, nx=40, ny=8, shared=True, tol=1e-10,
             max_iter=60),
        # Load sequences with different materials on one beam, advanced together.
        dict(name="dynamics_batch", kind="dynamics", nx=100, ny=10, nz=10, sequences=16, steps=1, max_inner=60),
        # Training of the warm-start network: an epoch's minibatches, then the weights back.
        dict(name="mlp_train", kind="mlp", width=256, layers=3, outputs=64, batch=512, updates=32, train=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _beam(rng, most):
    """Cells of a beam of about up to `most` cells, aspect 2 to 12, any remainder."""
    cells = math.exp(rng.uniform(math.log(40), math.log(most)))
    aspect = math.exp(rng.uniform(math.log(2.0), math.log(12.0)))
    ny = max(2, int(round((cells / aspect) ** (1.0 / 3.0))))
    nz = max(2, ny + rng.choice((-1, 0, 0, 1)))
    nx = max(4, min(int(cells / (ny * nz)), most // (ny * nz)))
    return nx, ny, nz


def draw(rng):
    kind = rng.choice(("force", "force", "static", "static", "step", "step", "batch", "batch", "dynamics", "mlp"))
    if kind == "force":
        nx, ny, nz = _beam(rng, 78000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, order=rng.choice((10, 10, 10, 4)),
                    precision=rng.choice(("fp64", "fp32")), damped=rng.random() < 0.25)
    if kind == "static":
        nx, ny, nz = _beam(rng, 60000)
        budget = rng.choice((25, 50, 80))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, order=rng.choice((10, 10, 4)), tol=1e-10,
                    max_iter=20000 if nx * ny * nz <= 4000 else min(budget, 2 * nx))
    if kind == "step":
        nx, ny, nz = _beam(rng, 30000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, order=rng.choice((10, 10, 4)),
                    solver=rng.choice(("nesterov", "nesterov", "adamw")), precision=rng.choice(("fp64", "fp64", "fp32")),
                    steps=rng.choice((1, 2)), max_outer=rng.choice((1, 2)), max_inner=rng.choice((15, 30, 45)))
    if kind == "batch":
        if rng.random() < 0.5:
            return dict(kind=kind, instances=_log(rng, 4, 48), nx_max=rng.randint(12, 48), ny_max=rng.randint(2, 5),
                        layout=rng.randint(1, 1 << 20), shared=False, tol=1e-10, max_iter=20000)
        nx = rng.randint(10, 40)
        return dict(kind=kind, instances=_log(rng, 3, 64), nx=nx, ny=rng.randint(2, 7), shared=True, tol=1e-10,
                    max_iter=rng.randint(nx, int(1.5 * nx)))
    if kind == "dynamics":
        nx, ny, nz = _beam(rng, 6000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, sequences=_log(rng, 2, 20), steps=rng.choice((1, 2)),
                    max_inner=rng.choice((16, 24, 40)))
    return dict(kind=kind, width=16 * rng.randint(4, 24), layers=rng.randint(2, 4), outputs=16 * rng.randint(2, 8),
                batch=16 * _log(rng, 1, 64), updates=rng.choice((8, 16, 24)), train=rng.random() < 0.7)


# ------------------------------------------------------------------------------- the inputs


@functools.lru_cache(maxsize=8)
def _box(nx, ny, nz, order):
    return M.box_mesh(nx, ny, nz, order, 1.0, 1.0, 1.0)


def _mesh(r, nx, ny, nz, order, lx=1.0, ly=0.1, lz=0.1):
    """A beam with its inner corner nodes moved by up to a tenth of a cell."""
    gx, gy, gz, conn = _box(nx, ny, nz, order)
    xs = []
    inner = (gx > 1e-9) & (gx < 1 - 1e-9) & (gy > 1e-9) & (gy < 1 - 1e-9) & (gz > 1e-9) & (gz < 1 - 1e-9)
    for g, length, n in ((gx, lx, nx), (gy, ly, ny), (gz, lz, nz)):
        v = length * g + np.where(inner, (0.1 * length / n) * r.uniform(-1.0, 1.0, g.shape), 0.0)
        if order == 10:
            for k, (a, b) in enumerate(((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))):
                v[conn[:, 4 + k]] = 0.5 * (v[conn[:, a]] + v[conn[:, b]])
        xs.append(v)
    return xs, conn


def _tip_load(r, xs, lo=10.0, hi=1000.0):
    x = xs[0]
    fixed = np.nonzero(x < 1e-9)[0].astype(np.int32)
    tip = np.nonzero(x > x.max() - 1e-9)[0]
    d = r.standard_normal(3)
    d *= r.uniform(lo, hi) / (np.linalg.norm(d) * len(tip))
    f = np.zeros((len(x), 3))
    f[tip] = d
    return fixed, f.ravel()


def _material(r):
    return float(np.exp(r.uniform(np.log(3e6), np.log(3e7)))), float(r.uniform(0.25, 0.4))


def _layout(case):
    """Cells along and across each beam of an uneven batch."""
    r = np.random.default_rng(case["layout"])
    return [(int(r.integers(8, case["nx_max"] + 1)), int(r.integers(2, case["ny_max"] + 1)))
            for _ in range(case["instances"])]


def _inputs(case, seed):
    """Everything that is random about a case, from the seed alone (host arrays)."""
    r = np.random.default_rng([seed, 77])
    kind = case["kind"]
    if kind == "mlp":
        dims = [6] + [case["width"]] * case["layers"] + [case["outputs"]]
        n = sum(a * b + b for a, b in zip(dims[:-1], dims[1:]))
        p = np.concatenate([r.uniform(-1, 1, a * b + b) / math.sqrt(a) for a, b in zip(dims[:-1], dims[1:])])
        x = r.uniform(-1, 1, (case["updates"], case["batch"], 6))
        mix = r.standard_normal((6, case["outputs"])) / np.arange(1, case["outputs"] + 1)
        t = np.sin(x @ mix)
        return dict(dims=dims, n=n, params=p.astype(np.float32), x=x.astype(np.float32), t=t.astype(np.float32))
    if kind == "batch":
        meshes, fixed, loads, e_mod, nu = [], [], [], [], []
        if case["shared"]:
            xs, conn = _mesh(r, case["nx"], case["ny"], case["ny"], 10)
            meshes.append((*xs, conn))
        else:
            for nx, ny in _layout(case):
                xs, conn = _mesh(r, nx, ny, ny, 10, 0.1 * ny, 0.01 * ny, 0.01 * ny)
                meshes.append((*xs, conn))
        for i in range(case["instances"]):
            xs = meshes[0 if case["shared"] else i][:3]
            fx, f = _tip_load(r, xs, 1.0, 500.0)
            e, n = float(np.exp(r.uniform(np.log(1e6), np.log(1e8)))), float(r.uniform(0.2, 0.45))
            fixed.append(fx)
            loads.append(f)
            e_mod.append(e)
            nu.append(n)
        if case["shared"]:
            meshes = meshes * case["instances"]
        u0 = None
        if case["shared"]:  # a smooth guess, zero at the clamped face, as a predictor gives it
            x = meshes[0][0]
            shape = np.stack([np.sin(0.5 * np.pi * x), x * x, 1 - np.cos(0.5 * np.pi * x)], 1)
            u0 = np.stack([shape * (1e-3 * r.standard_normal(3)) for _ in range(case["instances"])]).ravel()
        return dict(meshes=meshes, fixed=fixed, loads=loads, E=np.array(e_mod), nu=np.array(nu), u0=u0)
    xs, conn = _mesh(r, case["nx"], case["ny"], case["nz"], case.get("order", 10))
    fixed, f = _tip_load(r, xs, 10.0, 100.0)
    e_mod, nu = _material(r)
    d = dict(xs=xs, conn=conn, fixed=fixed, f=f, E=e_mod, nu=nu)
    n = len(xs[0])
    if kind == "force":
        # a bent and twisted beam (strains of some per cent) with a little noise, and velocities
        amp, ph = r.uniform(0.005, 0.02, 3), r.uniform(0, 2 * np.pi, 3)
        twist = r.uniform(-0.2, 0.2)
        x, y, z = xs
        k = np.pi * r.uniform(0.5, 1.5)
        ux = amp[0] * np.sin(k * x + ph[0]) + 2 * (y - 0.05) * amp[1]
        uy = amp[1] * np.sin(k * x + ph[1]) - twist * x * (z - 0.05)
        uz = amp[2] * np.sin(k * x + ph[2]) + twist * x * (y - 0.05)
        noise = 0.01 / max(case["nx"], 10)
        d["at"] = [v + u + noise * 0.1 * r.standard_normal(n) for v, u in zip(xs, (ux, uy, uz))]
        d["v"] = (0.1 * r.standard_normal((n, 3)) + np.stack([uy, uz, ux], 1)).ravel() if case["damped"] else None
        d["eta"], d["lam_d"] = (float(r.uniform(50, 200)), float(r.uniform(50, 200))) if case["damped"] else (0.0, 0.0)
    if kind == "step":
        d["f_var"] = d["f"]
        g = np.zeros((n, 3))
        g[:, 2] = -r.uniform(0.5, 1.0) * 9.81 * RHO * 0.01 / n  # dead weight, equal per node
        d["f"] = g.ravel()
        d["omega"], d["phase"] = float(2 * np.pi * r.uniform(3, 8)), float(r.uniform(0.5, 1.5))
    if kind == "dynamics":
        s = case["sequences"]
        d["E"] = np.exp(r.uniform(np.log(3e6), np.log(3e7), s))
        d["nu"] = r.uniform(0.25, 0.4, s)
        d["omega"], d["phase"] = float(2 * np.pi * 5), float(r.uniform(0.0, 1.0))
    return d


def _alpha(case, e_mod, nu, dt):
    """A stable gradient step for the step Hessian M/dt + dt K of this mesh and material."""
    h = max(1.0 / case["nx"], 0.1 / case["ny"], 0.1 / case["nz"])
    stiff = e_mod * h * (1 - nu) / ((1 + nu) * (1 - 2 * nu))
    return 0.3 / (dt * 8.0 * stiff)


STEP_RHO = 1e8
DT = 1e-3
ADAMW = dict(lr=2e-4, beta1=0.9, beta2=0.999, eps=1e-2, weight_decay=1e-4, lr_decay=0.998)


# ------------------------------------------------------------------------------- the state


class _Device:
    """A device array of the library as __cuda_array_interface__; keeps the array's owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (int(ptr), False),
                                         "version": 3, "strides": None}


def _view(owner, ptr, *shape):
    return torch.as_tensor(_Device(owner, ptr, shape), device=DEV)


def _element(d, order, eta=0.0, lam_d=0.0, mass=False, e_mod=None, nu=None):
    xs, conn = d["xs"], d["conn"]
    el = (T.GPU_FEAT10_Data if order == 10 else T.GPU_FEAT4_Data)(conn.shape[0], len(xs[0]))
    el.Initialize()
    el.SetNodalFixed(d["fixed"])
    el.SetExternalForce(d["f"])
    el.Setup(*(T.Quadrature.t10() if order == 10 else T.Quadrature.t4()), *xs, conn)
    el.SetDensity(RHO)
    el.SetDamping(eta, lam_d)
    el.SetSVK(d["E"] if e_mod is None else e_mod, d["nu"] if nu is None else nu)
    el.CalcDnDuPre()
    if mass:
        el.CalcMassMatrix()
        el.CalcConstraintData()
        el.ConvertToCSR_ConstraintJacT()
    return el


def _positions(el):
    return [_view(el, p, el.n_coef) for p in (el.GetX12DevicePtr(), el.GetY12DevicePtr(), el.GetZ12DevicePtr())]


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "force":
        el = _element(d, case["order"], d["eta"], d["lam_d"])
        el.SetForcePrecision(case["precision"])
        for v, a in zip(_positions(el), d["at"]):
            v.copy_(torch.as_tensor(a))
        s["v"] = torch.as_tensor(d["v"], device=DEV) if case["damped"] else None
        s["el"], s["d_v"] = el, s["v"].data_ptr() if case["damped"] else None
        s["f"] = _view(el, el.GetInternalForceDevicePtr(), 3 * el.n_coef)
    elif kind == "static":
        el = _element(d, case["order"])
        s["el"], s["solver"] = el, T.LinearStaticSolver(el, case["tol"], case["max_iter"])
        s["x"] = _positions(el)
    elif kind == "step":
        el = _element(d, case["order"], mass=True)
        el.SetForcePrecision(case["precision"])
        if case["solver"] == "nesterov":
            solver = T.SyncedNesterovSolver(el, el.get_n_constraint())
            solver.Setup()
            solver.SetParameters(T.SyncedNesterovParams(_alpha(case, d["E"], d["nu"], DT), STEP_RHO, 0.0, 0.0,
                                                        case["max_outer"], case["max_inner"], DT))
        else:
            solver = T.SyncedAdamWSolver(el, el.get_n_constraint())
            solver.Setup()
            solver.SetParameters(T.SyncedAdamWParams(ADAMW["lr"], ADAMW["beta1"], ADAMW["beta2"], ADAMW["eps"],
                                                     ADAMW["weight_decay"], ADAMW["lr_decay"], 0.0, 0.0, STEP_RHO,
                                                     case["max_outer"], case["max_inner"], DT, 10))
        s.update(el=el, solver=solver, x=_positions(el), f=d["f"], f_var=d["f_var"], omega=d["omega"], phase=d["phase"])
    elif kind == "batch":
        b = T.BatchedLinearStaticSolver(d["meshes"], T.TYPE_T10, shared=case["shared"])
        b.SetMaterial(d["E"], d["nu"])
        b.SetNodalFixed(d["fixed"])
        b.SetExternalForce(d["loads"])
        if d["u0"] is not None:
            b.SetInitialGuess(d["u0"])
        s["batch"], s["u"] = b, _view(b, b.DevicePtrs()["u"], 3 * b.n_nodes)
    elif kind == "dynamics":
        el = _element(d, 10, mass=True, e_mod=float(d["E"][0]), nu=float(d["nu"][0]))
        el.SetExternalForce(np.zeros(3 * el.n_coef))
        el.AddGravity(0.0, 0.0, -9.81)
        b = T.BatchedDynamics(el, case["sequences"])
        b.SetMaterial(d["E"], d["nu"])
        alpha = np.array([_alpha(case, e, n, DT) for e, n in zip(d["E"], d["nu"])])
        b.SetParameters(T.SyncedNesterovParams(float(alpha.min()), STEP_RHO, 0.0, 0.0, 1, case["max_inner"], DT), 0.0)
        b.SetStepSizes(alpha)
        b.SetLoad(d["f"], 1.0, d["omega"], d["phase"])
        b.SetRestart(True)
        p, n = b.DevicePtrs(), el.n_coef
        s.update(el=el, dyn=b, out={k: _view(b, p[k], case["sequences"], 3 * n if k == "v" else n) for k in "xyzv"})
    else:
        net = T.WarmStartMLP(d["dims"], max_batch=max(128, (case["batch"] + 127) // 128 * 128))
        net.SetParams(d["params"])
        s.update(net=net, p0=d["params"], x=torch.as_tensor(d["x"], device=DEV), t=torch.as_tensor(d["t"], device=DEV))
        s["y"] = torch.empty(d["t"].shape, dtype=torch.float32, device=DEV)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------- one pass


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "force":
        s["el"].ComputeInternalForce(s["d_v"])
        s["el"].GetInternalForceDevicePtr()
        return s["f"]
    if kind == "static":
        s["el"].ResetPositions()
        s["solver"].Solve()
        return s["x"]
    if kind == "step":
        s["el"].ResetPositions()
        s["el"].SetExternalForce(s["f"])
        s["solver"].Setup()
        s["solver"].RunSteps(case["steps"], s["f_var"], 1.0, s["omega"], s["phase"])
        return s["x"]
    if kind == "batch":
        s["batch"].Solve(case["tol"], case["max_iter"])
        return s["u"]
    if kind == "dynamics":
        s["dyn"].Reset()
        for _ in range(case["steps"]):
            s["dyn"].Step()
        return s["out"]
    net, x, t, batch = s["net"], s["x"], s["t"], case["batch"]
    if case["train"]:
        net.SetParams(s["p0"])
        for k in range(case["updates"]):
            net.TrainStep(x[k].data_ptr(), t[k].data_ptr(), batch)
        return net.GetParams()
    for k in range(case["updates"]):
        net.Forward(x[k].data_ptr(), batch, s["y"][k].data_ptr())
    return s["y"]


# ------------------------------------------------------------------------------- the least work


def _counts(nx, ny, nz, order):
    n, e = M.box_counts(nx, ny, nz, order)
    return n, e


def _iterations(nx, ny, nz):
    """CG iterations to 1e-10 on a beam of that many cells, about (965 at 10x2x2, 3471 at 40x8x8)."""
    return int(700 + 350 * max(ny, nz))


def _force_flops(order):
    """F, the stress and the nodal forces of an element, per quadrature point about 300 multiply-adds (TET10)."""
    return 5 * 600 if order == 10 else 250


def _tangent_flops(order):
    """K p of an element: the strain of p, the stress and the nodal forces, about 200 multiply-adds a point (TET10)."""
    return 5 * 400 if order == 10 else 160


def work(case):
    """Inputs read once and outputs written once; arithmetic of every evaluation that the method makes."""
    kind = case["kind"]
    if kind == "mlp":
        dims = [6] + [case["width"]] * case["layers"] + [case["outputs"]]
        w = sum(a * b + b for a, b in zip(dims[:-1], dims[1:]))
        rows = case["batch"] * case["updates"]
        return {"bytes": rows * 4 * (6 + case["outputs"]) + w * 4 * (2 if case["train"] else 1),
                "flops": 2.0 * w * rows * (3 if case["train"] else 1)}
    if kind == "batch":
        if case["shared"]:
            n, e = _counts(case["nx"], case["ny"], case["ny"], 10)
            return {"bytes": e * 40 + n * 24 + case["instances"] * n * 72,
                    "flops": case["instances"] * e * case["max_iter"] * _tangent_flops(10)}
        n, e = np.sum([_counts(nx, ny, ny, 10) for nx, ny in _layout(case)], axis=0)
        products = sum(_counts(nx, ny, ny, 10)[1] * _iterations(nx, ny, ny) for nx, ny in _layout(case))
        return {"bytes": int(e) * 40 + int(n) * 96, "flops": products * _tangent_flops(10)}
    order = case.get("order", 10)
    n, e = _counts(case["nx"], case["ny"], case["nz"], order)
    mesh = e * order * 4 + n * 24
    if kind == "force":
        return {"bytes": mesh + n * 48 + (n * 24 if case["damped"] else 0),
                "flops": e * _force_flops(order) * (1.4 if case["damped"] else 1.0)}
    if kind == "static":
        iters = min(case["max_iter"], _iterations(case["nx"], case["ny"], case["nz"]))
        return {"bytes": mesh + n * 48, "flops": iters * e * _tangent_flops(order)}
    evaluations = case["steps"] * case["max_inner"] * case.get("max_outer", 1) * case.get("sequences", 1)
    return {"bytes": mesh + n * 48 * case.get("sequences", 1), "flops": evaluations * e * _force_flops(order)}


# ------------------------------------------------------------------------------- the exact answer
# The same method in 64 bits with plain torch operations: gradients per quadrature point, forces and
# products by einsum, vectors by ordinary arithmetic.


def _rule(order):
    if order == 4:
        return np.array([[0.25] * 4]), np.array([1.0 / 6.0])
    a, b = 0.5, 1.0 / 6.0
    pts = np.array([[0.25] * 4, [a, b, b, b], [b, a, b, b], [b, b, a, b], [b, b, b, a]])
    return pts, np.array([-0.8, 0.45, 0.45, 0.45, 0.45]) / 6.0


def _shape(order):
    """Shape functions (Q, A) and their derivatives by xi (Q, A, 3) at the rule's points."""
    pts, w = _rule(order)
    dl = np.array([[-1.0, -1.0, -1.0], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
    if order == 4:
        return pts, np.broadcast_to(dl, (1, 4, 3)).copy(), w
    edges = ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))
    n = np.concatenate([pts * (2 * pts - 1), np.stack([4 * pts[:, i] * pts[:, j] for i, j in edges], 1)], 1)
    g = [(4 * pts[:, i] - 1)[:, None] * dl[i] for i in range(4)]
    g += [4 * (pts[:, i, None] * dl[j] + pts[:, j, None] * dl[i]) for i, j in edges]
    return n, np.stack(g, 1), w


class _Body:
    """Element geometry of one mesh (or several joined) in 64 bits on the device."""

    def __init__(self, xs, conn, lam, mu):
        order = conn.shape[1]
        n, dn, w = (torch.as_tensor(v, dtype=torch.float64, device=DEV) for v in _shape(order))
        self.x0 = torch.as_tensor(np.stack(xs, 1), dtype=torch.float64, device=DEV)
        self.conn = torch.as_tensor(conn, device=DEV).long()
        self.flat = self.conn.reshape(-1)
        rel = self.x0[self.conn] - self.x0[self.conn[:, :1]]
        jac = torch.einsum("eai,qaj->eqij", rel, dn)
        self.g = torch.einsum("qaj,eqji->eqai", dn, torch.linalg.inv(jac)).contiguous()
        self.dv = torch.linalg.det(jac) * w
        self.n = n
        self.eye = torch.eye(3, dtype=torch.float64, device=DEV)
        self.lam = torch.as_tensor(lam, dtype=torch.float64, device=DEV).reshape(-1, 1)
        self.mu = torch.as_tensor(mu, dtype=torch.float64, device=DEV).reshape(-1, 1)

    def _sum(self, fe):
        out = torch.zeros_like(self.x0)
        return out.index_add_(0, self.flat, fe.reshape(-1, 3))

    def _grad(self, u):
        return torch.einsum("eai,eqaj->eqij", u[self.conn] - u[self.conn[:, :1]], self.g)

    def force(self, u, v=None, eta=0.0, lam_d=0.0, lam=None, mu=None):
        lam, mu = (self.lam if lam is None else lam), (self.mu if mu is None else mu)
        h = self._grad(u)
        ht = h.transpose(-1, -2)
        e = 0.5 * (h + ht + ht @ h)
        s = (lam * e.diagonal(dim1=-2, dim2=-1).sum(-1))[..., None, None] * self.eye + 2 * (mu[..., None, None] * e)
        f = h + self.eye
        if v is not None:
            fd = self._grad(v)
            ed = 0.5 * (fd.transpose(-1, -2) @ f + f.transpose(-1, -2) @ fd)
            s = s + 2 * eta * ed + lam_d * ed.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None] * self.eye
        return self._sum(torch.einsum("eqij,eqaj->eai", (f @ s) * self.dv[..., None, None], self.g))

    def product(self, p, lam=None, mu=None):
        """The tangent at the reference configuration times p."""
        lam, mu = (self.lam if lam is None else lam), (self.mu if mu is None else mu)
        h = self._grad(p)
        s = (lam * h.diagonal(dim1=-2, dim2=-1).sum(-1))[..., None, None] * self.eye
        s = (s + mu[..., None, None] * (h + h.transpose(-1, -2))) * self.dv[..., None, None]
        return self._sum(torch.einsum("eqij,eqaj->eai", s, self.g))

    def mass(self, w):
        at = torch.einsum("qa,eai->eqi", self.n, w[self.conn]) * (RHO * self.dv)[..., None]
        return self._sum(torch.einsum("qa,eqi->eai", self.n, at))


def _lame(e_mod, nu):
    e_mod, nu = np.asarray(e_mod, float), np.asarray(nu, float)
    return e_mod * nu / ((1 + nu) * (1 - 2 * nu)), e_mod / (2 * (1 + nu))


def _cg(apply, f, free, iters, u=None, group=None, groups=1):
    """CG on the free DOFs, each group of nodes (instance) with its own scalars, as far as 64 bits go."""
    group = torch.zeros(len(f), dtype=torch.long, device=DEV) if group is None else group

    def dot(a, b):
        return torch.zeros(groups, dtype=torch.float64, device=DEV).index_add_(0, group, (a * b).sum(1))

    free = free[:, None]
    f = f * free
    u = torch.zeros_like(f) if u is None else u * free
    r = f - apply(u) * free
    p = r.clone()
    rr = dot(r, r)
    least = 1e-32 * dot(f, f)
    for k in range(iters):
        if k % 100 == 99 and not bool((rr > least).any()):
            break
        q = apply(p) * free
        a = torch.where(rr > least, rr / dot(p, q), 0.0)[group][:, None]
        u = u + a * p
        r = r - a * q
        new = dot(r, r)
        p = r + torch.where(rr > least, new / rr, 0.0)[group][:, None] * p
        rr = new
    return u


def _steps(case, d, body, lam, mu, e_mod, nu, sequence=False):
    """The implicit steps of the first-order solvers at fixed counts."""
    n = len(body.x0)
    f_base = torch.as_tensor(d["f"], device=DEV).reshape(-1, 3)
    f_var = f_base
    if sequence:
        f_base = body.mass(torch.tensor([0.0, 0.0, -9.81], dtype=torch.float64, device=DEV).expand(n, 3))
    else:
        f_var = torch.as_tensor(d["f_var"], device=DEV).reshape(-1, 3)
    held = torch.zeros((n, 1), dtype=torch.float64, device=DEV)
    held[torch.as_tensor(d["fixed"], device=DEV).long()] = 1.0
    u = torch.zeros((n, 3), dtype=torch.float64, device=DEV)
    v, v_prev, mult = torch.zeros_like(u), torch.zeros_like(u), torch.zeros_like(u)
    alpha = _alpha(case, e_mod, nu, DT)
    for step in range(case["steps"]):
        f_ext = f_base + math.sin(d["omega"] * (step + 1) * DT + d["phase"]) * f_var
        u_prev = u

        def gradient(w):
            at = u_prev + DT * w
            return (body.mass((w - v_prev) / DT) + body.force(at, lam=lam, mu=mu) - f_ext
                    + DT * held * (mult + STEP_RHO * at))

        for _ in range(case.get("max_outer", 1)):
            if case.get("solver", "nesterov") == "nesterov":
                vk, vkm1, t, beta = v, v, 1.0, 0.0
                mom = 0
                betas = []
                for _ in range(case["max_inner"] + 1):
                    tn = 0.5 * (1 + math.sqrt(1 + 4 * t * t))
                    betas.append((t - 1) / tn)
                    t = tn
                for _ in range(case["max_inner"]):
                    y = vk + betas[mom] * (vk - vkm1)
                    g = gradient(y)
                    nxt = y - alpha * g
                    again = sequence and float((g * (nxt - vk)).sum()) > 0
                    mom = 0 if again else mom + 1
                    vkm1, vk = vk, nxt
                v = vk
            else:
                a = ADAMW
                g, m1, m2, lr = torch.zeros_like(v), torch.zeros_like(v), torch.zeros_like(v), a["lr"]
                for k in range(case["max_inner"]):
                    lr *= a["lr_decay"]
                    m1 = a["beta1"] * m1 + (1 - a["beta1"]) * g
                    m2 = a["beta2"] * m2 + (1 - a["beta2"]) * g * g
                    step_dir = (m1 / (1 - a["beta1"] ** (k + 2))) / ((m2 / (1 - a["beta2"] ** (k + 2))).sqrt() + a["eps"])
                    v = v - lr * (step_dir + a["weight_decay"] * v)
                    g = gradient(v)
            v_prev = v
            u = u_prev + DT * v
            mult = mult + STEP_RHO * DT * held * u
    return u, v


def _network(case, d):
    dims = d["dims"]
    w, b, o = [], [], 0
    p = torch.as_tensor(d["params"], device=DEV).double()
    for k, m in zip(dims[:-1], dims[1:]):
        w.append(p[o:o + k * m].reshape(m, k).clone().requires_grad_(True))
        b.append(p[o + k * m:o + k * m + m].clone().requires_grad_(True))
        o += k * m + m

    def forward(x):
        for i, (wi, bi) in enumerate(zip(w, b)):
            x = x @ wi.T + bi
            if i + 1 < len(w):
                x = torch.nn.functional.gelu(x)
        return x

    x, t = (torch.as_tensor(d[k], device=DEV).double() for k in "xt")
    if not case["train"]:
        with torch.no_grad():
            return torch.stack([forward(v) for v in x])
    opt = torch.optim.AdamW([*w, *b], lr=1e-3, betas=(0.9, 0.999), eps=1e-8, weight_decay=0.0)
    for xi, ti in zip(x, t):
        opt.zero_grad()
        torch.nn.functional.mse_loss(forward(xi), ti).backward()
        opt.step()
    return torch.cat([torch.cat([wi.detach().reshape(-1), bi.detach()]) for wi, bi in zip(w, b)])


def exact(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "mlp":
        return _network(case, d)
    if kind == "batch":
        k, off = case["instances"], 0
        n_of = [len(m[0]) for m in d["meshes"]]
        e_of = [len(m[3]) for m in d["meshes"]]
        lam, mu = _lame(d["E"], d["nu"])
        f = torch.as_tensor(np.concatenate(d["loads"]), device=DEV).reshape(-1, 3)
        group = torch.repeat_interleave(torch.arange(k, device=DEV), torch.tensor(n_of, device=DEV))
        free = torch.ones(len(f), dtype=torch.float64, device=DEV)
        conns = []
        for i, m in enumerate(d["meshes"]):
            free[torch.as_tensor(d["fixed"][i] + off, device=DEV).long()] = 0.0
            conns.append(m[3] + off)
            off += n_of[i]
        u0 = torch.as_tensor(d["u0"], device=DEV).reshape(-1, 3) if d["u0"] is not None else None
        if case["shared"]:
            body = _Body(d["meshes"][0][:3], d["meshes"][0][3], 0.0, 0.0)
            n = n_of[0]

            def apply(p):
                return torch.cat([body.product(p[i * n:(i + 1) * n], torch.as_tensor(lam[i], device=DEV).reshape(1, 1),
                                               torch.as_tensor(mu[i], device=DEV).reshape(1, 1)) for i in range(k)])
        else:
            body = _Body([np.concatenate([m[j] for m in d["meshes"]]) for j in range(3)], np.concatenate(conns),
                         np.repeat(lam, e_of), np.repeat(mu, e_of))
            apply = body.product
        return _cg(apply, f, free, case["max_iter"], u0, group, k).reshape(-1)
    if kind == "dynamics":
        if case["sequences"] * case["steps"] * case["max_inner"] > 1200:
            return None
        body = _Body(d["xs"], d["conn"], 0.0, 0.0)
        xs, vs = [], []
        for e, nu in zip(d["E"], d["nu"]):
            lam, mu = (torch.as_tensor(v, device=DEV).reshape(1, 1) for v in _lame(e, nu))
            u, v = _steps(case, d, body, lam, mu, float(e), float(nu), sequence=True)
            xs.append(u + body.x0)
            vs.append(v.reshape(-1))
        x = torch.stack(xs)
        return {"x": x[..., 0], "y": x[..., 1], "z": x[..., 2], "v": torch.stack(vs)}
    body = _Body(d["xs"], d["conn"], *_lame(d["E"], d["nu"]))
    if kind == "force":
        u = torch.as_tensor(np.stack(d["at"], 1), device=DEV) - body.x0
        v = torch.as_tensor(d["v"], device=DEV).reshape(-1, 3) if case["damped"] else None
        return body.force(u, v, d["eta"], d["lam_d"]).reshape(-1)
    if kind == "static":
        free = torch.ones(len(body.x0), dtype=torch.float64, device=DEV)
        free[torch.as_tensor(d["fixed"], device=DEV).long()] = 0.0
        f = torch.as_tensor(d["f"], device=DEV).reshape(-1, 3)
        u = _cg(body.product, f, free, case["max_iter"])
    else:
        u, _ = _steps(case, d, body, body.lam, body.mu, d["E"], d["nu"])
    x = u + body.x0
    return [x[:, 0], x[:, 1], x[:, 2]]
