"""Moment sets of a caller's own that end within a degree (n between those of two
orders), which the instances of whole orders do not fit: the fused kernels with
runtime tile counts, Mn and PPn, with the Gaunt table and with products.

The vectors are the moments of known multipliers, which the solves must give
back: the stopping test leaves a gradient of at most tol ||u / u_0||, and the
multipliers' error is that over the Hessian's smallest eigenvalue (above 1e-3
for these).  The two tables sum the same Hessian, so their solves agree as two
layouts do (tol = 1e-6 as in the layouts' tests: at 1e-8 the line search of some
vectors is decided by the last bit of f).
"""
import ctypes as C

import numpy as np
import pytest

import closures_b200 as cb

pytestmark = pytest.mark.gpu


class _Cut:
    """The first n moments of an order's tables."""

    def __init__(self, order, n, Q, gaunt):
        self.full = cb.Angular(order, Q, gaunt)
        f = self.full
        self._a = type(f._a)()
        C.memmove(C.byref(self._a), C.byref(f._a), C.sizeof(f._a))
        self.n = self._a.n = n
        self.w, self.p = f.w, f.p[:, :n].copy()
        if gaunt:
            off, idx, val = [0], [], []
            for i in range(n):
                for j in range(n):
                    r = slice(f.gaunt_off[i * f.n + j], f.gaunt_off[i * f.n + j + 1])
                    idx.extend(f.gaunt_idx[r])
                    val.extend(f.gaunt_val[r])
                    off.append(len(idx))
            self.arrays = (np.array(off, np.int32), np.array(idx, np.int32), np.array(val))
            self._a.gaunt_nnz = len(idx)
            self._a.gaunt_off = self.arrays[0].ctypes.data_as(C.POINTER(C.c_int))
            self._a.gaunt_idx = self.arrays[1].ctypes.data_as(C.POINTER(C.c_int))
            self._a.gaunt_val = self.arrays[2].ctypes.data_as(C.POINTER(C.c_double))


def _vectors(a, count, closure, seed):
    rng = np.random.default_rng(seed)
    alpha = 0.3 * rng.uniform(-1.0, 1.0, (count, a.n))
    if closure == cb.CL_PPN:
        alpha[:, 0] += 1.0
        k = 0.5 * alpha @ a.p.T
        G = k + np.sqrt(k * k + 1e-10)
    else:
        G = np.exp(alpha @ a.p.T)
    return (G * a.w) @ a.p, alpha


@pytest.mark.parametrize("order,n", [(2, 4), (2, 5), (3, 7), (3, 8), (3, 9), (4, 12), (5, 16), (5, 20), (6, 25)])
@pytest.mark.parametrize("closure", [cb.CL_MN, cb.CL_PPN])
def test_partial_orders(order, n, closure):
    count, out = 150, []
    for gaunt in (1, 0):
        a = _Cut(order, n, 2 * order + 8, gaunt)
        u, alpha = _vectors(a, count, closure, order * 100 + n)
        ctx = cb.Context.for_batches(a, cb.make_options(moment_type=closure, tol=1e-6))
        ug, ag = u.copy(), cb.isotropic_alpha(n, count, moment_type=closure)
        it, reg, st = ctx.solve_batch(ug, ag)
        ctx.close()
        assert (st == 0).all() and (reg == 0).all()
        unorm = np.linalg.norm(u / u[:, :1], axis=1)
        assert np.all(np.linalg.norm(ug - u, axis=1) / u[:, 0] <= 1.001e-6 * unorm)
        assert np.max(np.abs(ag - alpha)) < 1e-3 * np.max(unorm)
        out.append((ug, it))
    assert np.array_equal(out[0][1], out[1][1])
    assert np.max(np.abs(out[0][0] - out[1][0]) / out[1][0][:, :1]) < 1e-10
