"""The straight-sided element paths against the oracle, at the sizes where their tiles and
launches change: less than one tile, exactly one, a ragged last tile, the resident launch's
limit and beyond it; and the meshes that must not take them.

Bars: forces and products are sums of products of the same data in another order; the
geometry of a straight element is its corners', whose distance from the per-point one is the
rounding of the coordinates, 1e-16 |x| / h.  With h >= 1/200 of the beam that is under 1e-13,
times a few tens of additions: 1e-11 for products of random vectors.  Converged solves differ
by the tolerance 1e-10 times the beam's condition: 1e-7."""
import numpy as np
import pytest
import scipy.sparse as sp

import tlfea_b200 as T
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


@pytest.mark.parametrize("cells,order", [((3, 1, 1), 10), ((4, 2, 2), 10), ((9, 3, 2), 10), ((23, 5, 4), 10),
                                         ((3, 1, 1), 4), ((31, 7, 5), 4)])
def test_linear_solve_on_the_linear_operator(cells, order):
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


# 592 resident tiles of 128 elements: 75,776 elements; on either side of it
@pytest.mark.parametrize("cells", [(120, 10, 10), (130, 10, 10)])
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


def test_curved_and_degenerate_meshes_keep_the_general_path():
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
