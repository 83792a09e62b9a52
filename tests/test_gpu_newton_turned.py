"""Angular tables of a caller's own, Gaunt orders 3-6: azimuths turned by a part
of their spacing keep phi -> phi + pi and lose phi -> -phi, so they run as
direction pairs, in both launch shapes and with the screening pass; a table
with neither symmetry runs one direction at a time.

Turning the quadrature turns the problem: the moments R u on the turned table
have the solution R alpha of u on the library's table.  Bounds as for the
library's layouts: same decisions, multipliers to 1e-7 (rounding times the
Hessian's condition), moments to 1e-10.
"""
import ctypes as C

import numpy as np
import pytest

import closures_b200 as cb

pytestmark = pytest.mark.gpu


def _turned(order, Q, part):
    """The library's tables with every azimuth advanced by part * pi / Q, and
    the matrix R: basis values p(turned) = R p."""
    a = cb.Angular(order, Q, 1)
    d = part * np.pi / Q
    R = np.zeros((a.n2, a.n2))
    at = {}
    k = 0
    for l in range(2 * order + 1):
        for m in range(-l, l + 1, 2):
            at[l, m] = k
            k += 1
    for (l, m), k in at.items():
        c, s = np.cos(abs(m) * d), np.sin(abs(m) * d)
        R[k, k] = c
        if m != 0:
            R[k, at[l, -m]] = -s if m > 0 else s
    p = np.ctypeslib.as_array(a._a.p, shape=(a.nq, a.n2))
    p[:] = p @ R.T
    xi = np.ctypeslib.as_array(a._a.xi, shape=(a.nq,))
    eta = np.ctypeslib.as_array(a._a.eta, shape=(a.nq,))
    xi[:], eta[:] = xi * np.cos(d) - eta * np.sin(d), eta * np.cos(d) + xi * np.sin(d)
    # the Gaunt table holds on the turned directions as well
    off, idx, val = a.gaunt_off, a.gaunt_idx, a.gaunt_val
    for i, j in ((1, 2), (a.n - 1, a.n - 2), (a.n - 1, 1)):
        r = slice(off[i * a.n + j], off[i * a.n + j + 1])
        assert np.max(np.abs(p[:, i] * p[:, j] - p[:, idx[r]] @ val[r])) < 1e-12
    return a, R[:a.n, :a.n]


def _solve(ctx, u):
    ur, ar = u.copy(), cb.isotropic_alpha(u.shape[1], len(u))
    it, reg, st = ctx.solve_batch(ur, ar)
    assert (st == 0).all()
    return ur, ar, it, reg


@pytest.mark.parametrize("order,Q,count", [(3, 10, 300), (4, 12, 33), (5, 14, 257), (6, 16, 4737)])
def test_turned_tables_run_as_pairs(order, Q, count):
    lib = cb.Angular(order, Q, 1)
    u0 = cb.sample_moment_vectors(lib, count, seed=order, s_range=(0.1, 1.0))[0]
    opts = cb.make_options(tol=1e-6)
    ctx = cb.Context.for_batches(lib, opts)
    u_ref, a_ref, it_ref, reg_ref = _solve(ctx, u0)
    ctx.close()
    a, R = _turned(order, Q, 0.3)
    for warps, contraction in ((None, None), (8, cb.CL_CONTRACT_PAIRS), (4, cb.CL_CONTRACT_PAIRS),
                               (8, cb.CL_CONTRACT_SINGLE)):
        ctx = cb.Context.for_batches(a, opts)
        assert ctx.tuning()["newton_contraction"] == "pairs"
        if warps:
            ctx.set_launch_shape(warps, contraction)
        ur, ar, it, reg = _solve(ctx, np.ascontiguousarray(u0 @ R.T))
        ctx.close()
        assert np.array_equal(it, it_ref) and np.array_equal(reg, reg_ref)
        assert np.max(np.abs(ur - u_ref @ R.T) / np.abs(u_ref[:, :1])) < 1e-10
        assert np.max(np.abs(ar - a_ref @ R.T)) < 1e-7 * np.max(np.abs(a_ref))


@pytest.mark.parametrize("order,Q", [(3, 10), (6, 16)])
def test_turned_grid_screens(order, Q):
    """Grid steps of the turned table, screening pass included, as pairs and
    one direction at a time."""
    a, R = _turned(order, Q, 0.3)
    nx, ny = 21, 18
    cells = (nx + 4) * (ny + 4)
    u = cb.sample_moment_vectors(cb.Angular(order, Q, 1), cells, seed=7, s_range=(0.05, 0.3))[0] @ R.T
    grid = cb.cl_grid(nx, ny, 2, 0, 0.0, 0.0, 2.0)
    out = []
    for contraction in (cb.CL_CONTRACT_PAIRS, cb.CL_CONTRACT_SINGLE):
        ctx = cb.Context(grid, cb.make_options(tol=1e-6, contraction=contraction), a, np.ones(cells),
                         0.5 * np.ones(cells), u, cb.isotropic_alpha(a.n, cells))
        for _ in range(3):
            ctx.step(1e-3, 0.1, 0.1)
        out.append((ctx.get_state(), ctx.last_iterations(), ctx.stats()))
        ctx.close()
    ((m1, a1), it1, s1), ((m2, a2), it2, _) = out
    assert s1["screen_evals"] > 0
    assert np.array_equal(it1, it2)
    assert np.max(np.abs(m1 - m2) / np.abs(m2[:, :, :1])) < 1e-10


def test_no_symmetry_runs_single():
    a = cb.Angular(3, 10, 1)
    np.ctypeslib.as_array(a._a.w, shape=(a.nq,))[3] *= 1.0 + 1e-9
    ctx = cb.Context.for_batches(a, cb.make_options(tol=1e-6))
    assert ctx.tuning()["newton_contraction"] == "single"
    u = cb.sample_moment_vectors(cb.Angular(3, 10, 1), 40, seed=1, s_range=(0.1, 1.0))[0]
    _solve(ctx, u)
    ctx.close()
