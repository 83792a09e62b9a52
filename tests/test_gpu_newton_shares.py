"""How K1 shares out its vectors, and its per-slot logic at every moment count.

A launch with fewer vectors than slots spreads them over the CTAs; a larger
one hands the rest out from the work counter.  Each vector's solve is its own,
so a batch solved at once, in two pieces, or in reverse order gives the same
bits.  The counts straddle the edges: one vector, one more than the CTAs, one
more than the slots.  The first vectors are held to the oracle: equal decisions
and moments to 1e-10 (the suite's bound where both oracle builds agree).
"""
import numpy as np
import pytest

import closures_b200 as cb
import pyoracle as oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,Q,gaunt,count", [
    (1, 20, 1, 149), (2, 20, 0, 1), (2, 20, 0, 149), (3, 20, 1, 4737), (3, 20, 0, 149), (4, 20, 1, 149),
    (4, 20, 0, 33), (5, 20, 1, 149), (6, 30, 1, 1), (6, 30, 1, 4737)])
def test_shares_and_oracle(order, Q, gaunt, count):
    a = cb.Angular(order, Q, gaunt)
    u, _ = cb.sample_moment_vectors(a, count, seed=order, s_range=(0.1, 2.0))
    a0 = cb.isotropic_alpha(a.n, count)
    ctx = cb.Context.for_batches(a, cb.make_options(tol=1e-6))

    def solve(rows):
        ur, ar = np.ascontiguousarray(u[rows]), np.ascontiguousarray(a0[rows])
        it, reg, st = ctx.solve_batch(ur, ar)
        assert (st == 0).all()
        return ur, ar, it, reg

    whole = solve(np.arange(count))
    for x, y in zip(solve(np.arange(count)[::-1]), whole):
        assert np.array_equal(x[::-1], y)
    cut = count // 3 + 1
    for x, y in zip(solve(np.arange(cut)), whole):
        assert np.array_equal(x, y[:cut])
    k = min(count, 48)
    uo, ao = u[:k].copy(), a0[:k].copy()
    it_o, reg_o, st_o = oracle_lib.opt_batch(order, Q, gaunt, uo, ao, tol=1e-6)
    assert (st_o == 0).all()
    assert np.array_equal(whole[2][:k], it_o) and np.array_equal(whole[3][:k], reg_o)
    assert np.max(np.abs(whole[0][:k] - uo) / np.abs(uo[:, :1])) < 1e-10
    ctx.close()
