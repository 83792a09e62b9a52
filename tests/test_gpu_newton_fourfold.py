"""The fourfold-direction layout of the Gaunt orders 3-6 against one direction
at a time, in both launch shapes.

One row stands for phi, phi + pi, -phi and pi - phi; the quadrature sizes give
(Q/2)^2 rows: less than a chunk of 32, one more than a chunk, an odd number,
whole chunks.  Both layouts evaluate the same sums in another order, so the
solves take the same decisions; the multipliers may differ by rounding times
the Hessian's condition (1e-15 x 1e6 at these vectors; held to 1e-7), moments
by the suite's 1e-10.
"""
import numpy as np
import pytest

import closures_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warps", [8, 4])
@pytest.mark.parametrize("order,Q,count", [(3, 10, 17), (3, 20, 1), (4, 12, 300), (4, 32, 9), (5, 14, 33),
                                           (5, 20, 4737), (6, 16, 8), (6, 30, 257)])
def test_fourfold_equals_single(order, Q, count, warps):
    a = cb.Angular(order, Q, 1)
    u, _ = cb.sample_moment_vectors(a, count, seed=order, s_range=(0.1, 1.0))
    a0 = cb.isotropic_alpha(a.n, count)
    out = []
    for contraction in (cb.CL_CONTRACT_PAIRS, cb.CL_CONTRACT_SINGLE):
        ctx = cb.Context.for_batches(a, cb.make_options(tol=1e-6, contraction=contraction))
        if contraction == cb.CL_CONTRACT_PAIRS:
            ctx.set_launch_shape(warps, contraction)
        ur, ar = u.copy(), a0.copy()
        it, reg, st = ctx.solve_batch(ur, ar)
        assert (st == 0).all()
        out.append((ur, ar, it, reg))
        ctx.close()
    (u1, a1, it1, reg1), (u2, a2, it2, reg2) = out
    assert np.array_equal(it1, it2) and np.array_equal(reg1, reg2)
    assert np.max(np.abs(u1 - u2) / np.abs(u2[:, :1])) < 1e-10
    assert np.max(np.abs(a1 - a2)) < 1e-7 * np.max(np.abs(a2))
