"""Gaunt tables longer than a well-resolved quadrature's: order 6 with Q = 2N = 12,
whose extended basis is dependent on its directions, has 26 entry groups instead
of 12.  Beside 32 slots there is no room to stage it; the layout stays the
folded one, with 16 slots.  Against the oracle's direct products: the same
sums, so the same decisions and the suite's 1e-10.
"""
import numpy as np
import pytest

import closures_b200 as cb
import pyoracle as oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,Q,closure,count", [(6, 12, cb.CL_MN, 700), (6, 12, cb.CL_MN, 5), (6, 12, cb.CL_PPN, 700),
                                                   (5, 10, cb.CL_MN, 300)])
@pytest.mark.parametrize("contraction", [cb.CL_CONTRACT_PAIRS, cb.CL_CONTRACT_SINGLE])
def test_coarsest_quadrature(order, Q, closure, count, contraction):
    a = cb.Angular(order, Q, 1)
    u, _ = cb.sample_moment_vectors(a, count, seed=order, s_range=(0.1, 0.5))
    a0 = cb.isotropic_alpha(a.n, count, moment_type=closure)
    ctx = cb.Context.for_batches(a, cb.make_options(moment_type=closure, tol=1e-6, contraction=contraction))
    pairs = closure == cb.CL_MN and contraction == cb.CL_CONTRACT_PAIRS
    assert ctx.tuning()["newton_contraction"] == ("pairs" if pairs else "single")
    if pairs:
        for warps in (8, 4):
            ctx.set_launch_shape(warps, contraction)
            assert order < 6 or ctx.tuning()["newton_warps"] == 4
    ug, ag = u.copy(), a0.copy()
    it_g, reg_g, st_g = ctx.solve_batch(ug, ag)
    ctx.close()
    uo, ao = u.copy(), a0.copy()
    it_o, reg_o, st_o = oracle_lib.opt_batch(order, Q, 0, uo, ao, moment_type=closure, tol=1e-6)
    assert (st_g == 0).all() and np.array_equal(it_g, it_o) and np.array_equal(reg_g, reg_o)
    assert np.max(np.abs(ug - uo) / uo[:, :1]) < 1e-10
