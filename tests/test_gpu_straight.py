"""The straight-sided element paths against the oracle, at the sizes where their tiles and
launches change: tiles whole and ragged, each block width of the resident launches, their
limit and beyond it; and the meshes that must not take them.

Bars: forces and products are sums of products of the same data in another order; the
geometry of a straight element is its corners', whose distance from the per-point one is the
rounding of the coordinates, 1e-16 |x| / h.  With h >= 1/200 of the beam that is under 1e-13,
times a few tens of additions: 1e-11 for products of random vectors.  Converged solves differ
by the tolerance 1e-10 times the beam's condition: 1e-7."""
from pathlib import Path

import numpy as np
import pytest
import scipy.sparse as sp

import tlfea_b200 as T
from tlfea_b200 import _capi as capi
from oracle import oracle as O
from tlfea_b200 import mesh as M

from .helpers import box, lame, make_element, perturb, rel

pytestmark = pytest.mark.gpu
LAM, MU = lame()


def jitter(x, y, z, conn, scale, seed=3):
    """Corner nodes moved, mid-edge nodes at the midpoints."""
    r = np.random.default_rng(seed)
    out = []
    for v in (x, y, z):
        v = v + scale * r.uniform(-1, 1, v.shape)
        if conn.shape[1] == 10:
            for k, (a, b) in enumerate(((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))):
                v[conn[:, 4 + k]] = 0.5 * (v[conn[:, a]] + v[conn[:, b]])
        out.append(v)
    return out


def oracle_k(x, y, z, conn, f, fixed):
    g, dj = O.dndu_pre(x, y, z, conn)
    off, cols, vals = O.stiffness(x, y, z, conn, g, dj, LAM, MU)
    kv, fb = O.apply_bcs(off, cols, vals, f, fixed)
    return off, cols, kv, fb


# the linear operator from two tiles of quadratic elements on: two with a ragged end (252 elements), three whole
# ones (384), three and 22 with ragged ends; one tile and linear elements keep the assembled K
@pytest.mark.parametrize("cells,order", [((3, 1, 1), 10), ((4, 2, 2), 10), ((7, 3, 2), 10), ((8, 4, 2), 10),
                                         ((9, 3, 2), 10), ((23, 5, 4), 10), ((3, 1, 1), 4), ((31, 7, 5), 4)])
def test_linear_solve_from_the_reference_configuration(cells, order):
    import torch

    x, y, z, conn = box(*cells, order)
    fixed, f, _ = M.cantilever_loads(x, y, z, (1.0, 5.0, -20.0))
    x, y, z = jitter(x, y, z, conn, 0.05 / max(cells[0], 10 * cells[1]))
    off, cols, kv, fb = oracle_k(x, y, z, conn, f, fixed)
    u_ref, _, _, _ = O.cg(off, cols, kv, fb, 1e-12, 20000)
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f, mass=False)
    s = T.LinearStaticSolver(el, 1e-10, 20000)
    s.Solve()
    u = (np.stack(el.RetrievePositionToCPU()) - np.stack([x, y, z])).T.ravel()
    assert s.GetLastResidual() < 1e-10 and 0 < s.GetLastIterCount() < 20000
    assert rel(u, u_ref) < 1e-7
    xv = torch.tensor(np.random.default_rng(2).standard_normal(f.size), dtype=torch.float64, device="cuda")
    yv = torch.empty_like(xv)
    torch.cuda.synchronize()
    s.Apply(xv.data_ptr(), yv.data_ptr())
    torch.cuda.synchronize()
    K = sp.csr_matrix((kv, cols, off), shape=(f.size, f.size))
    assert rel(yv.cpu().numpy(), K @ xv.cpu().numpy()) < 1e-11
    o2, c2, v2 = s.RetrieveStiffnessCSRToCPU()
    assert np.array_equal(o2, off) and np.array_equal(c2, cols) and rel(v2, kv) < 1e-11
    # the second solve starts from the deformed positions: K at those, not the linear operator
    s.Solve()
    x1 = np.stack([x, y, z]) + u.reshape(-1, 3).T
    g, dj = O.dndu_pre(x, y, z, conn)
    off, cols, vals = O.stiffness(*x1, conn, g, dj, LAM, MU)
    kv, fb = O.apply_bcs(off, cols, vals, f, fixed)
    u2_ref, _, _, _ = O.cg(off, cols, kv, fb, 1e-12, 20000)
    u2 = (np.stack(el.RetrievePositionToCPU()) - x1).T.ravel()
    assert rel(u2, u2_ref) < 1e-6
    del s
    el.Destroy()


@pytest.mark.parametrize("change", ["material", "mooney", "damping", "reference", "fixed"])
def test_operator_of_the_last_solve_outlives_changes_to_the_element(change):
    """Apply and the stiffness matrix are the last solve's, whatever the element was given since."""
    import torch

    x, y, z, conn = box(9, 3, 2, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (1.0, 5.0, -20.0))
    x, y, z = jitter(x, y, z, conn, 0.002)
    off, cols, kv, _ = oracle_k(x, y, z, conn, f, fixed)
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f, mass=False)
    s = T.LinearStaticSolver(el, 1e-10, 20000)
    s.Solve()
    if change == "material":
        el.SetSVK(3e6, 0.2)
    elif change == "mooney":
        el.SetMooneyRivlin(1e6, 2e5, 5e7)
    elif change == "damping":
        el.SetDamping(10.0, 5.0)
    elif change == "reference":
        el.UpdatePositions(1.1 * x, y, z)
        el.CalcDnDuPre()
        det = el.RetrieveDetJToCPU()
    else:
        el.UpdateNodalFixed(fixed[:3])
    xv = torch.tensor(np.random.default_rng(2).standard_normal(f.size), dtype=torch.float64, device="cuda")
    yv = torch.empty_like(xv)
    torch.cuda.synchronize()
    s.Apply(xv.data_ptr(), yv.data_ptr())
    torch.cuda.synchronize()
    K = sp.csr_matrix((kv, cols, off), shape=(f.size, f.size))
    assert rel(yv.cpu().numpy(), K @ xv.cpu().numpy()) < 1e-11
    o2, c2, v2 = s.RetrieveStiffnessCSRToCPU()
    assert np.array_equal(o2, off) and np.array_equal(c2, cols) and rel(v2, kv) < 1e-11
    if change == "reference":  # and the element's geometry is the new one
        assert np.array_equal(el.RetrieveDetJToCPU(), det)
        el.ResetPositions()
        el.ComputeInternalForce()
        assert np.linalg.norm(el.RetrieveInternalForceToCPU()) < 1e-6
    del s
    el.Destroy()


# the resident solve's blocks of 512 (a tile per SM), 256 (two) and 128 threads: 24, 197, 282, 563 tiles; beyond
# its 592 tiles
@pytest.mark.parametrize("cells", [(16, 8, 4), (42, 10, 10), (60, 10, 10), (120, 10, 10), (130, 10, 10)])
def test_resident_and_phased_forms_agree_at_a_fixed_count(cells):
    x, y, z, conn = box(*cells, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (0.0, 3.0, -100.0))
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f, mass=False)
    out = []
    for operator in ("auto", "assembled"):
        s = T.LinearStaticSolver(el, 1e-10, 37)
        s.SetOperator(operator)
        s.Solve()
        assert s.GetLastIterCount() == 37
        out.append((np.stack(el.RetrievePositionToCPU()) - np.stack([x, y, z])).T.ravel())
        el.ResetPositions()
        del s
    assert rel(out[0], out[1]) < 1e-9
    el.Destroy()


# the smallest and the largest such budget, between them the one that showed the difference; 80 and
# 1000 lie outside: the linear operator, whose iterates agree to 1e-13 of the positions (80) and, where
# the solve converges, to the tolerance
@pytest.mark.parametrize("budget", [80, 81, 100, 999, 1000])
def test_stopped_solves_return_the_iterates_of_the_assembled_operator(budget):
    x, y, z, conn = box(24, 4, 4, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (0.0, 3.0, -100.0))
    x, y, z = jitter(x, y, z, conn, 0.002)
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f, mass=False)
    out = []
    for operator in ("auto", "assembled"):
        s = T.LinearStaticSolver(el, 1e-10, budget)
        s.SetOperator(operator)
        s.Solve()
        assert s.GetLastIterCount() == budget
        out.append(np.stack(el.RetrievePositionToCPU()))
        el.ResetPositions()
        del s
    assert np.array_equal(out[0], out[1]) == (81 <= budget <= 999)
    if budget == 80:
        assert rel(out[0], out[1]) < 1e-9
    el.Destroy()


def test_stopped_solve_of_a_large_mesh_returns_the_recorded_iterate():
    """150 iterations at 108,192 elements, every 499th node, as the per-point operator gave them on a B200:
    rounding in another order moves this iterate by 2e-8."""
    x, y, z, conn = box(92, 14, 14, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (0.0, 3.0, -100.0))
    x, y, z = jitter(x, y, z, conn, 7e-4, 1)
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f, mass=False)
    s = T.LinearStaticSolver(el, 1e-10, 150)
    s.Solve()
    want = np.load(Path(__file__).parent / "golden" / "stopped_cg_t10.npz")["positions"]
    assert rel(np.stack(el.RetrievePositionToCPU())[:, ::499], want) < 1e-9
    del s
    el.Destroy()


def test_phased_solve_converges_to_the_assembled_solution():
    """Beyond the resident limit (610 tiles), at the bar of converged solves."""
    x, y, z, conn = box(130, 10, 10, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (1.0, 3.0, -100.0))
    x, y, z = jitter(x, y, z, conn, 7e-4)
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f, mass=False)
    out = []
    for operator in ("auto", "assembled"):
        s = T.LinearStaticSolver(el, 1e-10, 20000)
        s.SetOperator(operator)
        s.Solve()
        assert s.GetLastResidual() < 1e-10 and s.GetLastIterCount() < 20000
        out.append(np.stack(el.RetrievePositionToCPU()) - np.stack([x, y, z]))
        el.ResetPositions()
        del s
    assert rel(out[0], out[1]) < 1e-7
    el.Destroy()


def test_curved_meshes_keep_the_general_path():
    x, y, z, conn = box(6, 2, 2, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (0.0, 0.0, -20.0))
    r = np.random.default_rng(5)
    edge = np.unique(conn[:, 4:])
    xc, yc, zc = x.copy(), y.copy(), z.copy()
    for v in (xc, yc, zc):
        v[edge] += 1e-3 * r.uniform(-1, 1, edge.size)  # curved edges
    off, cols, kv, fb = oracle_k(xc, yc, zc, conn, f, fixed)
    u_ref, _, _, _ = O.cg(off, cols, kv, fb, 1e-12, 20000)
    el = make_element(xc, yc, zc, conn, fixed=fixed, f_ext=f, mass=False)
    s = T.LinearStaticSolver(el, 1e-10, 20000)
    s.Solve()
    u = (np.stack(el.RetrievePositionToCPU()) - np.stack([xc, yc, zc])).T.ravel()
    assert rel(u, u_ref) < 1e-7
    del s
    el.Destroy()


def test_zero_load_no_iterations_and_breakdown():
    x, y, z, conn = box(4, 2, 2, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (0.0, 0.0, -20.0))
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=0 * f, mass=False)
    s = T.LinearStaticSolver(el, 1e-10, 100)
    s.Solve()
    assert s.GetLastIterCount() == 0 and s.GetLastResidual() == 0.0
    el.SetExternalForce(f)
    s0 = T.LinearStaticSolver(el, 1e-10, 0)
    s0.Solve()
    assert s0.GetLastIterCount() == 0 and s0.GetLastResidual() == 1.0
    assert np.array_equal(np.stack(el.RetrievePositionToCPU()), np.stack([x, y, z]))
    # a material without stiffness: p.Kp = 0, the reference's breakdown
    el.SetSVK(0.0, 0.3)
    sb = T.LinearStaticSolver(el, 1e-10, 100)
    sb.Solve()
    assert sb.GetLastIterCount() == 100 and sb.GetLastResidual() == 1.0
    del s, s0, sb
    el.Destroy()


# ---------------------------------------------------------------- internal force
# 6 elements; three whole tiles (384); a ragged last tile; more tiles than resident blocks (610)
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 1e-5)])  # the element tests' bars
@pytest.mark.parametrize("cells,order", [((1, 1, 1), 10), ((8, 4, 2), 10), ((9, 3, 2), 10), ((130, 10, 10), 10),
                                         ((1, 1, 1), 4), ((8, 4, 2), 4), ((31, 7, 5), 4)])
def test_internal_force_of_straight_elements(cells, order, prec, tol):
    import torch

    x, y, z, conn = box(*cells, order)
    x, y, z = jitter(x, y, z, conn, 0.05 / max(cells[0], 10 * cells[1]))
    el = make_element(x, y, z, conn, eta=2.0e3, lamd=5.0e2, mass=False)
    el.SetForcePrecision(prec)
    xs = perturb(x, y, z, 0.02 / max(cells[0], 10 * cells[1]), 6)
    el.UpdatePositions(*xs)
    g, dj = O.dndu_pre(x, y, z, conn)
    el.ComputeInternalForce()
    assert rel(el.RetrieveInternalForceToCPU(), O.force(*xs, conn, g, dj, LAM, MU)) < tol
    v = np.random.default_rng(2).standard_normal(3 * len(x)) * 0.1
    dv = torch.tensor(v, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    el.ComputeInternalForce(dv.data_ptr())
    f = el.RetrieveInternalForceToCPU()
    assert rel(f, O.force(*xs, conn, g, dj, LAM, MU, 2.0e3, 5.0e2, v)) < tol
    el.ComputeInternalForce(dv.data_ptr())
    assert np.array_equal(el.RetrieveInternalForceToCPU(), f)
    el.Destroy()


def with_a_flat_element(x, y, z, conn):
    """One more element, of no volume: four corners of a cell's face, mid-edge nodes at the midpoints."""
    order = conn.shape[1]
    face = [int(np.argmin(np.abs(x - a) + np.abs(y - b) + np.abs(z))) for a, b in
            ((0.0, 0.0), (x.max(), 0.0), (x.max(), y.max()), (0.0, y.max()))]
    new, xs = list(face), [x, y, z]
    if order == 10:
        for a, b in ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3)):
            new.append(len(xs[0]))
            xs = [np.append(v, 0.5 * (v[face[a]] + v[face[b]])) for v in xs]
    return (*xs, np.concatenate([conn, np.array([new], conn.dtype)]))


@pytest.mark.parametrize("order", [10, 4])
def test_degenerate_element_keeps_the_general_path(order):
    """The default is the gradient stream's result bit for bit, and the oracle's."""
    x, y, z, conn = with_a_flat_element(*box(9, 3, 2, order))
    el = make_element(x, y, z, conn, mass=False)
    xs = perturb(x, y, z, 1e-3, 6)
    el.UpdatePositions(*xs)
    el.ComputeInternalForce()
    f = el.RetrieveInternalForceToCPU()
    el.SetLaunchConfig("tma")
    el.ComputeInternalForce()
    assert np.array_equal(f, el.RetrieveInternalForceToCPU())
    g, dj = O.dndu_pre(x, y, z, conn)
    assert rel(f, O.force(*xs, conn, g, dj, LAM, MU)) < 1e-10
    el.Destroy()


@pytest.mark.parametrize("ulps,straight", [(0, True), (3, True), (6, False), (1e6, False)])
def test_straight_sided_up_to_four_units_in_the_last_place(ulps, straight):
    """One mid-edge node moved by units in the last place of its element's coordinates, which lie in
    [0.5, 1): 2.2e-16 times the largest of them a unit."""
    x, y, z, conn = box(9, 3, 2, 10)
    x = 0.5 + 0.5 * x * (1 - 2 ** -30)
    e = len(conn) - 1
    big = x[conn[e]].max()
    for k, (a, b) in enumerate(((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))):
        x[conn[:, 4 + k]] = 0.5 * (x[conn[:, a]] + x[conn[:, b]])
    x[conn[e, 4]] += ulps * 2.220446049250313e-16 * big
    el = make_element(x, y, z, conn, mass=False)
    xs = perturb(x, y, z, 1e-3, 6)
    el.UpdatePositions(*xs)
    el.ComputeInternalForce()
    f = el.RetrieveInternalForceToCPU()
    el.SetLaunchConfig("tma")
    el.ComputeInternalForce()
    assert np.array_equal(f, el.RetrieveInternalForceToCPU()) == (not straight)
    g, dj = O.dndu_pre(x, y, z, conn)
    assert rel(f, O.force(*xs, conn, g, dj, LAM, MU)) < 1e-10
    el.Destroy()


def test_points_in_another_order_keep_the_general_path():
    """The rule with its points permuted: the same sums, by the per-point kernels."""
    from tlfea_b200 import quadrature as Q

    x, y, z, conn = box(9, 3, 2, 10)
    el = T.GPU_FEAT10_Data(conn.shape[0], len(x))
    el.Initialize()
    order = [3, 1, 0, 4, 2]
    el.Setup(*(np.ascontiguousarray(v[order]) for v in Q.t10()), x, y, z, conn)
    el.SetDensity(1000.0)
    el.SetDamping(0.0, 0.0)
    el.SetSVK(1e7, 0.3)
    el.CalcDnDuPre()
    xs = perturb(x, y, z, 1e-3, 6)
    el.UpdatePositions(*xs)
    el.ComputeInternalForce()
    f = el.RetrieveInternalForceToCPU()
    el.SetLaunchConfig("tma")
    el.ComputeInternalForce()
    assert np.array_equal(f, el.RetrieveInternalForceToCPU())
    g, dj = O.dndu_pre(x, y, z, conn)
    assert rel(f, O.force(*xs, conn, g, dj, LAM, MU)) < 1e-10
    el.Destroy()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_non_finite_positions_stay_in_their_elements(bad, prec):
    """The force is not finite at the nodes of the elements that hold the node, as from the gradient stream;
    a first-order solve from there reports it."""
    x, y, z, conn = box(9, 3, 2, 10)
    fixed, f_ext, _ = M.cantilever_loads(x, y, z, (10.0, 20.0, -50.0))
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f_ext)
    el.SetForcePrecision(prec)
    xs = perturb(x, y, z, 1e-3, 6)
    xs[1][conn[100, 5]] = bad
    el.UpdatePositions(*xs)
    finite = []
    for kernel in ("auto", "tma"):
        el.SetLaunchConfig(kernel)
        el.ComputeInternalForce()
        finite.append(np.isfinite(el.RetrieveInternalForceToCPU().reshape(-1, 3)).all(1))
    near = np.unique(conn[(conn == conn[100, 5]).any(1)])
    assert not finite[0][near].any() and np.array_equal(finite[0], finite[1])
    s = T.SyncedNesterovSolver(el, el.get_n_constraint())
    s.Setup()
    s.SetParameters(T.SyncedNesterovParams(1.0e-5, 1e8, 0.0, 0.0, 1, 8, 1.0e-3))
    with pytest.raises(T.TLFEAError, match="NONFINITE"):
        s.Solve()
    del s
    el.Destroy()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_default_force_kernel_can_be_chosen_again(prec):
    x, y, z, conn = box(9, 3, 2, 10)
    el = make_element(x, y, z, conn, mass=False)
    el.SetForcePrecision(prec)
    el.UpdatePositions(*perturb(x, y, z, 1e-3, 6))
    el.ComputeInternalForce()
    first = el.RetrieveInternalForceToCPU()
    out = []
    for kernel in ("tma", "auto"):
        el.SetLaunchConfig(kernel)
        el.ComputeInternalForce()
        out.append(el.RetrieveInternalForceToCPU())
    assert np.array_equal(out[1], first) and not np.array_equal(out[0], first)
    for bad in (-2, 4):
        with pytest.raises(T.TLFEAError):
            el.SetLaunchConfig(bad)
    el.Destroy()


def test_internal_force_beside_orphans_and_of_curved_elements():
    x, y, z, conn = box(5, 2, 2, 10)
    r = np.random.default_rng(5)
    xo, yo, zo = (np.concatenate([v, [7.0, 8.0]]) for v in (x, y, z))  # two nodes without elements
    edge = np.unique(conn[:, 4:])
    xc, yc, zc = x.copy(), y.copy(), z.copy()
    for v in (xc, yc, zc):
        v[edge] += 1e-3 * r.uniform(-1, 1, edge.size)
    for p in ((xo, yo, zo), (xc, yc, zc)):
        el = make_element(*p, conn, mass=False)
        xs = perturb(*p, 1e-3, 6)
        el.UpdatePositions(*xs)
        g, dj = O.dndu_pre(*p, conn)
        el.ComputeInternalForce()
        f = el.RetrieveInternalForceToCPU()
        assert rel(f, O.force(*xs, conn, g, dj, LAM, MU)) < 1e-10
        assert not f.reshape(-1, 3)[np.setdiff1d(np.arange(len(p[0])), conn)].any()
        el.Destroy()


# ---------------------------------------------------------------- first-order solvers
# one tile, whole tiles, a ragged last tile; 197 and 352 tiles: the resident launch's blocks of 192 threads (two
# tiles an SM) and of 128 (AdamW; Nesterov's phases); 610: beyond it (444 in FP64)
@pytest.mark.parametrize("kind,cells,order", [
    ("nesterov", (3, 2, 2), 10), ("nesterov", (8, 4, 2), 10), ("nesterov", (9, 3, 2), 10),
    ("nesterov", (31, 3, 2), 4), ("nesterov", (130, 10, 10), 10), ("adamw", (9, 3, 2), 10), ("adamw", (31, 3, 2), 4),
    ("nocoop", (8, 4, 2), 10), ("adamw", (130, 10, 10), 10), ("nesterov", (42, 10, 10), 10),
    ("nesterov", (75, 10, 10), 10), ("adamw", (42, 10, 10), 10), ("adamw", (75, 10, 10), 10),
    ("nocoop", (42, 10, 10), 10), ("nocoop", (75, 10, 10), 10), ("nesterov", (42, 10, 10), 4), ("adamw", (75, 10, 10), 4)])
def test_first_order_steps_on_straight_elements(kind, cells, order):
    from .test_gpu_solvers import ADAMW, E_MOD, _oracle_displacement_with_bar

    x, y, z, conn = box(*cells, order)
    fixed, f, _ = M.cantilever_loads(x, y, z, (10.0, 20.0, -50.0))
    if kind == "nesterov":
        params = (1.0e-5, 1e8, 0.0, 0.0, 2, 8, 1.0e-3)
        s_cls, p = T.SyncedNesterovSolver, T.SyncedNesterovParams(*params)
    else:
        a = list(ADAMW)
        a[0], a[3], a[6], a[7], a[8], a[9], a[10] = 1e-3, 1.0, 0.0, 0.0, 1e4, 2, 8
        params = tuple(a)
        s_cls = T.SyncedAdamWSolver if kind == "adamw" else T.SyncedAdamWNocoopSolver
        p = T.SyncedAdamWParams(*params)
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f)
    s = s_cls(el, el.get_n_constraint())
    s.Setup()
    s.SetParameters(p)
    for _ in range(2):
        s.Solve()
    assert s.GetStats()["inner_iters_total"] == 16
    # both AdamW solvers take the same steps at a fixed count
    disp, bar = _oracle_displacement_with_bar(x, y, z, conn, E_MOD, fixed, f, "nesterov" if kind == "nesterov" else
                                              "adamw", params, 2)
    assert rel(np.stack(el.RetrievePositionToCPU()) - np.stack([x, y, z]), disp) < bar
    del s
    el.Destroy()


@pytest.mark.parametrize("point", [(0.25, 0.25, 0.25), (0.1, 0.2, 0.3), (0.0, 0.0, 1.0)])
@pytest.mark.parametrize("prec,tol", [("fp64", 1e-10), ("fp32", 1e-5)])
def test_mass_of_linear_elements_follows_the_point(point, prec, tol):
    """One quadrature point anywhere in the element: Nesterov, AdamW and a batch of sequences against the
    persistent kernel, which takes the shape functions at the point (the solvers' and the forces' bars)."""
    x, y, z, conn = box(31, 3, 2, 4)
    fixed, f, _ = M.cantilever_loads(x, y, z, (10.0, 20.0, -50.0))
    nesterov = T.SyncedNesterovParams(1.0e-5, 1e8, 0.0, 0.0, 2, 8, 1.0e-3)
    adamw = T.SyncedAdamWParams(2e-4, 0.9, 0.999, 1.0, 1e-4, 0.995, 0.0, 0.0, 1e4, 2, 8, 1e-3, 10)

    def element():
        el = T.GPU_FEAT4_Data(conn.shape[0], len(x))
        el.Initialize()
        el.SetNodalFixed(fixed)
        el.SetExternalForce(f)
        el.Setup(*(np.array([v]) for v in point), np.array([1.0 / 6.0]), x, y, z, conn)
        el.SetDensity(1000.0)
        el.SetDamping(0.0, 0.0)
        el.SetSVK(1e7, 0.3)
        el.CalcDnDuPre()
        el.CalcMassMatrix()
        el.CalcConstraintData()
        el.ConvertToCSR_ConstraintJacT()
        el.SetForcePrecision(prec)
        return el

    def moved(cls, params, mode):
        el = element()
        s = cls(el, el.get_n_constraint())
        s.Setup()
        s.SetParameters(params)
        s.SetMode(mode)
        for _ in range(2):
            s.Solve()
        out = np.stack(el.RetrievePositionToCPU()) - np.stack([x, y, z])
        del s
        el.Destroy()
        return out

    ref = moved(T.SyncedNesterovSolver, nesterov, "persistent")
    assert rel(moved(T.SyncedNesterovSolver, nesterov, "auto"), ref) < tol
    assert rel(moved(T.SyncedAdamWSolver, adamw, "auto"), moved(T.SyncedAdamWSolver, adamw, "persistent")) < tol
    if prec == "fp64":  # (sequences have FP64 forces)
        el = element()
        b = T.BatchedDynamics(el, 2)
        b.SetMaterial(np.array([1e7, 1e7]), np.array([0.3, 0.3]))
        b.SetParameters(nesterov, 0.0)
        for _ in range(2):
            b.Step(T.BatchedDynamics.WARM_PREVIOUS)
        assert rel(np.stack(b.RetrievePositions(1)) - np.stack([x, y, z]), ref) < tol
        b.Destroy()
        el.Destroy()


# 9 tiles resident, 610 in launches whose graphs are kept from solve to solve
@pytest.mark.parametrize("cells", [(9, 3, 2), (130, 10, 10)])
def test_density_changed_between_solves(cells):
    """The second solve from rest equals a fresh solver's at the new density, bit for bit."""
    x, y, z, conn = box(*cells, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (10.0, 20.0, -50.0))
    out = []
    for first in (1000.0, 3000.0):
        el = make_element(x, y, z, conn, rho=first, fixed=fixed, f_ext=f)
        s = T.SyncedNesterovSolver(el, el.get_n_constraint())
        s.SetParameters(T.SyncedNesterovParams(1.0e-5, 1e8, 0.0, 0.0, 2, 8, 1.0e-3))
        for rho in ((first, 3000.0) if first != 3000.0 else (3000.0,)):
            el.SetDensity(rho)
            el.CalcMassMatrix()
            el.ResetPositions()
            s.Setup()
            s.Solve()
        out.append(np.stack(el.RetrievePositionToCPU()))
        del s
        el.Destroy()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("damped", [False, True])
def test_density_and_damping_changed_between_steps_of_sequences(damped):
    x, y, z, conn = box(9, 3, 2, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (10.0, 20.0, -50.0))
    last = (3000.0, 2.0e3 if damped else 0.0)
    out = []
    for first in ((1000.0, 1.0e3 if damped else 0.0), last):
        el = make_element(x, y, z, conn, rho=first[0], fixed=fixed, f_ext=f, eta=first[1])
        b = T.BatchedDynamics(el, 3)
        b.SetMaterial(np.array([1e7, 3e6, 2e7]), np.array([0.3, 0.25, 0.35]))
        b.SetParameters(T.SyncedNesterovParams(1.0e-6, 1e8, 0.0, 0.0, 2, 8, 1.0e-3), 0.0)
        for rho, eta in ((first, last) if first != last else (last,)):
            el.SetDensity(rho)
            el.SetDamping(eta, 0.0)
            el.CalcMassMatrix()
            b.Reset()
            b.Step()
        out.append([np.stack(b.RetrievePositions(s)) for s in range(3)])
        b.Destroy()
        el.Destroy()
    assert np.array_equal(out[0], out[1])


# the resident launch in FP32: blocks of 512, 256 and 128 threads (up to 592 tiles); beyond it
@pytest.mark.parametrize("kind,cells", [("nesterov", (9, 3, 2)), ("nesterov", (42, 10, 10)), ("nesterov", (130, 10, 10)),
                                        ("adamw", (42, 10, 10)), ("adamw", (110, 10, 10))])
def test_first_order_fp32_forces_on_straight_elements(kind, cells):
    """Element forces in FP32 against the oracle: the solvers' bar for FP32 forces, 1e-4 of the
    displacement."""
    from .test_gpu_solvers import ADAMW, E_MOD, _oracle_displacement_with_bar

    x, y, z, conn = box(*cells, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (10.0, 20.0, -50.0))
    params = (1.0e-5, 1e8, 0.0, 0.0, 2, 8, 1.0e-3)
    if kind == "adamw":
        a = list(ADAMW)
        a[0], a[3], a[6], a[7], a[8], a[9], a[10] = 1e-3, 1.0, 0.0, 0.0, 1e4, 2, 8
        params = tuple(a)
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f)
    el.SetForcePrecision("fp32")
    s = (T.SyncedNesterovSolver if kind == "nesterov" else T.SyncedAdamWSolver)(el, el.get_n_constraint())
    s.Setup()
    s.SetParameters((T.SyncedNesterovParams if kind == "nesterov" else T.SyncedAdamWParams)(*params))
    s.Solve()
    disp, _ = _oracle_displacement_with_bar(x, y, z, conn, E_MOD, fixed, f, kind, params, 1)
    assert rel(np.stack(el.RetrievePositionToCPU()) - np.stack([x, y, z]), disp) < 1e-4
    del s
    el.Destroy()


def test_fp32_forces_in_the_solver_are_no_further_off_than_per_point():
    """60 Nesterov iterations with FP32 forces against the FP64 solver on the per-point kernels: the mean
    distance over four meshes is no larger than the per-point FP32 kernels'."""
    err = {"auto": [], "persistent": []}
    for seed in range(4):
        x, y, z, conn = box(20, 4, 4, 10)
        fixed, f, _ = M.cantilever_loads(x, y, z, (50.0, 0.0, 0.0))
        x, y, z = jitter(x, y, z, conn, 0.0025, seed)

        def run(mode, prec):
            el = make_element(x, y, z, conn, fixed=fixed, f_ext=f)
            el.SetForcePrecision(prec)
            s = T.SyncedNesterovSolver(el, el.get_n_constraint())
            s.Setup()
            s.SetParameters(T.SyncedNesterovParams(5.0e-5, 1e8, 0.0, 0.0, 1, 60, 1.0e-3))
            s.SetMode(mode)
            s.Solve()
            out = np.stack(el.RetrievePositionToCPU()) - np.stack([x, y, z])
            del s
            el.Destroy()
            return out

        exact = run("persistent", "fp64")
        assert np.linalg.norm(exact) < 1e-2 * np.linalg.norm(np.stack([x, y, z]))  # a stable step size
        for mode, e in err.items():
            e.append(rel(run(mode, "fp32"), exact))
    assert np.mean(err["auto"]) <= np.mean(err["persistent"]), err


# ---------------------------------------------------------------- batches
# the group sizes of the launch (1, 2, 4, 8 sequences a block) and their remainders
@pytest.mark.parametrize("n,cells,order", [(1, (8, 4, 2), 10), (2, (9, 3, 2), 10), (5, (3, 2, 2), 10),
                                           (9, (9, 3, 2), 10), (17, (4, 2, 2), 10), (3, (31, 3, 2), 4)])
def test_sequences_on_straight_elements(n, cells, order):
    from .test_gpu_dynamics import _batch, _mesh, _oracle_with_bar

    x, y, z, conn, fixed, f, _ = _mesh(cells, order, (10.0, 20.0, -50.0))
    r = np.random.default_rng(n)
    E, nu = np.exp(r.uniform(np.log(1e6), np.log(2e7), n)), r.uniform(0.2, 0.4, n)
    params = (1.0e-6, 1e8, 0.0, 0.0, 2, 8, 1.0e-3)
    el, b = _batch(x, y, z, conn, fixed, f, E, nu, params)
    for _ in range(2):
        b.Step(T.BatchedDynamics.WARM_PREVIOUS)
    X0 = np.stack([x, y, z])
    for s in sorted({0, n // 2, n - 1}):
        disp, vel, bx, bv = _oracle_with_bar(x, y, z, conn, E[s], nu[s], fixed, [f, f], params)
        assert rel(np.stack(b.RetrievePositions(s)) - X0, disp[1]) < bx
        assert rel(b.RetrieveVelocity(s), vel[1]) < bv
    b.Destroy()
    el.Destroy()


# tiles that two or more instances share, instances of many tiles, single instances; on one
# mesh, groups of several sizes with remainders
@pytest.mark.parametrize("shared,n,order", [(False, 1, 10), (False, 7, 10), (False, 23, 10), (False, 9, 4),
                                            (True, 2, 10), (True, 13, 10), (True, 33, 10), (True, 5, 4)])
def test_batched_operator_and_iterates_on_straight_elements(shared, n, order):
    """Products against the oracle's matrix; iterates after 20 steps at the batch tests' bar, for
    quadratic elements (a 48-node mesh of linear ones is at its solution by then, where the
    oracle's own iterate moves by 1e-8 when its matrix does by 1e-16)."""
    import torch

    from .test_gpu_batch import _oracle_kbc

    insts = [M.random_beam(300 + (0 if shared else i), nx_range=(2, 14), ny_range=(1, 4), order=order)
             for i in range(n)]
    r = np.random.default_rng(n)
    for d in insts:
        d.update(E=float(np.exp(r.uniform(np.log(1e6), np.log(1e9)))), nu=float(r.uniform(0.2, 0.45)),
                 f=d["f"] * r.uniform(0.5, 2.0))
    b = T.BatchedLinearStaticSolver([(d["x"], d["y"], d["z"], d["conn"]) for d in insts],
                                    T.TYPE_T10 if order == 10 else T.TYPE_T4, shared=shared)
    b.SetMaterial([d["E"] for d in insts], [d["nu"] for d in insts])
    b.SetNodalFixed([d["fixed"] for d in insts])
    b.SetExternalForce([d["f"] for d in insts])
    xs = [r.standard_normal(3 * len(d["x"])) for d in insts]
    xd = torch.tensor(np.concatenate(xs), dtype=torch.float64, device="cuda")
    yd = torch.empty_like(xd)
    torch.cuda.synchronize()
    b.Apply(xd.data_ptr(), yd.data_ptr())
    b.Solve(1e-300, 20)
    assert np.all(b.GetResults()[0] == 20)
    us, y, o = b.RetrieveDisplacement(), yd.cpu().numpy(), 0
    for k, (d, xv) in enumerate(zip(insts, xs)):
        off, cols, kv, fb = _oracle_kbc(d)
        assert rel(y[o:o + xv.size], O.spmv(off, cols, kv, xv)) < 1e-11
        if order == 10:
            assert rel(us[k], O.cg(off, cols, kv, fb, 0.0, 20)[0]) < 1e-9
        o += xv.size
    b.Destroy()


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("left", [1, 2, 3])  # of 33: up to a sixteenth the node phases run on the resident blocks
def test_instances_left_of_a_batch_iterate_as_in_a_full_one(shared, left):
    """The others have no load and are done at once; the iterates are the same bit for bit."""
    insts = [M.random_beam(300 + (0 if shared else i), nx_range=(6, 14), ny_range=(2, 3)) for i in range(33)]
    b = T.BatchedLinearStaticSolver([(d["x"], d["y"], d["z"], d["conn"]) for d in insts], T.TYPE_T10, shared=shared)
    b.SetMaterial([1e7 * (1 + 0.1 * i) for i in range(33)], [0.3] * 33)
    b.SetNodalFixed([d["fixed"] for d in insts])
    running = [0, 17, 32][:left]
    out = []
    for who in (range(33), running):
        b.SetExternalForce([d["f"] if i in who else 0 * d["f"] for i, d in enumerate(insts)])
        b.Solve(1e-300, 100)
        assert [b.GetResults()[0][i] for i in running] == [100] * left
        u = b.RetrieveDisplacement()
        out.append([u[i] for i in running])
    assert all(np.array_equal(p, q) for p, q in zip(*out))
    b.Destroy()


def test_batches_on_straight_elements_hold_one_set_of_buffers():
    """Against the same batch on a curved mesh, which runs the general kernels: a shared batch takes no more
    memory; sequences take less than 96 bytes a node more, which two records of 32 and at least one slot of 32
    a node would be beside the general buffers."""
    import torch

    x, y, z, conn = box(40, 8, 8, 10)
    yc = y.copy()
    edge = np.unique(conn[:, 4:])
    yc[edge] += 1e-4 * np.random.default_rng(5).uniform(-1, 1, edge.size)
    n = 64 * len(x)

    def used(create):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        b = create()
        took = free - torch.cuda.mem_get_info()[0]
        b.Destroy()
        return took

    shared, sequences = [], []
    for ys in (y, yc):
        el = make_element(x, ys, z, conn)
        shared.append(used(lambda: T.BatchedLinearStaticSolver([(x, ys, z, conn)] * 64, T.TYPE_T10, shared=True)))
        sequences.append(used(lambda: T.BatchedDynamics(el, 64)))
        el.Destroy()
    assert shared[0] <= shared[1]
    assert sequences[0] - sequences[1] < 96 * n


# ---------------------------------------------------------------- waits that run out
def late(fn, *args):
    """The call reports the error word of an expired wait, once."""
    with pytest.raises(T.TLFEAError, match="BUDGET_EXCEEDED"):
        fn(*args)


# static solves: resident (9 tiles), in launches per phase (610 tiles), on the assembled K; explicit steps
@pytest.mark.parametrize("cells,operator", [((9, 3, 2), "auto"), ((130, 10, 10), "auto"), ((9, 3, 2), "assembled")])
def test_static_solves_report_an_expired_wait(cells, operator):
    import torch

    x, y, z, conn = box(*cells, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (0.0, 3.0, -100.0))
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f, mass=False)
    s = T.LinearStaticSolver(el, 1e-10, 25)
    s.SetOperator(operator)
    capi.call("tlfea_test_expire_wait", el._handle())
    late(s.Solve)
    assert np.array_equal(np.stack(el.RetrievePositionToCPU()), np.stack([x, y, z]))
    v = torch.zeros(3 * len(x), dtype=torch.float64, device="cuda")
    w = torch.empty_like(v)
    torch.cuda.synchronize()
    if operator == "auto":  # (with the assembled operator K stands)
        with pytest.raises(T.TLFEAError, match="NOT_SETUP"):
            s.Apply(v.data_ptr(), w.data_ptr())
    s.Solve()
    assert s.GetLastIterCount() == 25
    if operator == "auto":
        capi.call("tlfea_test_expire_wait", el._handle())
        late(s.Apply, v.data_ptr(), w.data_ptr())
        s.Apply(v.data_ptr(), w.data_ptr())
    del s
    el.Destroy()


@pytest.mark.parametrize("cells", [(9, 3, 2), (130, 10, 10)])
def test_steps_report_an_expired_wait(cells):
    x, y, z, conn = box(*cells, 10)
    fixed, f, _ = M.cantilever_loads(x, y, z, (10.0, 20.0, -50.0))
    params = T.SyncedNesterovParams(1.0e-6, 1e8, 0.0, 0.0, 1, 8, 1.0e-3)
    el = make_element(x, y, z, conn, fixed=fixed, f_ext=f)
    s = T.SyncedNesterovSolver(el, el.get_n_constraint())
    s.Setup()
    s.SetParameters(params)
    capi.call("tlfea_test_expire_wait", el._handle())
    late(s.Solve)
    s.Solve()
    capi.call("tlfea_test_expire_wait", el._handle())
    late(s.RunSteps, 2)
    b = T.BatchedDynamics(el, 2)
    b.SetMaterial(np.array([1e7, 5e6]), np.array([0.3, 0.3]))
    b.SetParameters(params, 0.0)
    capi.call("tlfea_test_expire_wait", el._handle())
    late(b.Step)
    b.Step()
    b.Destroy()
    del s
    el.Destroy()


@pytest.mark.parametrize("mode,prec", [("phased", "fp64"), ("phased", "fp32"), ("persistent", "fp64"),
                                       ("persistent", "fp32")])
@pytest.mark.parametrize("shared", [False, True])
def test_batches_report_an_expired_wait(shared, mode, prec):
    import torch

    d = M.random_beam(300, nx_range=(6, 14), ny_range=(2, 4), order=10)
    b = T.BatchedLinearStaticSolver([(d["x"], d["y"], d["z"], d["conn"])] * 3, T.TYPE_T10, shared=shared)
    b.SetMaterial([1e7] * 3, [0.3] * 3)
    b.SetNodalFixed([d["fixed"]] * 3)
    b.SetExternalForce([d["f"]] * 3)
    b.SetMode(mode)
    b.SetPrecision(prec)
    capi.call("tlfea_test_expire_batch_wait", b._h)
    late(b.Solve, 1e-6, 2000)
    b.Solve(1e-6, 2000)
    assert not b.GetResults()[2].any()
    v = torch.zeros(3 * b.n_nodes, dtype=torch.float64, device="cuda")
    w = torch.empty_like(v)
    torch.cuda.synchronize()
    capi.call("tlfea_test_expire_batch_wait", b._h)
    late(b.Apply, v.data_ptr(), w.data_ptr())
    b.Destroy()


def test_elements_beyond_the_shared_page_have_words_of_their_own():
    """512 elements share a page of host words; the ones after it, and one in it, report for themselves."""
    x, y, z, conn = box(1, 1, 1, 4)
    crowd = [T.GPU_FEAT4_Data(conn.shape[0], len(x)) for _ in range(511)]
    for el in crowd:
        el.Initialize()
    els = [make_element(x, y, z, conn, mass=False) for _ in range(3)]
    for k in range(3):
        capi.call("tlfea_test_expire_wait", els[k]._handle())
        for j in range(3):
            if j == k:
                late(els[j].ComputeInternalForce)
            els[j].ComputeInternalForce()
    for el in crowd + els:
        el.Destroy()
