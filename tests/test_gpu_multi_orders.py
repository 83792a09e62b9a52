"""Mixed-order solves, a launch per order on streams of their own: every order's
results are those of a batch of its own, to the bit, for counts of none, one,
one more than the CTAs, and very uneven ones, in any order of the orders.
"""
import numpy as np
import pytest
import torch

import closures_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("orders,counts", [
    ([3], [1]), ([2, 4], [0, 149]), ([5, 1, 3, 2, 4], [1, 5000, 0, 149, 33]),
    ([1, 2, 3, 4, 5, 6, 2, 3], [7, 300, 1, 64, 2, 65, 1, 2000]), ([6, 1], [0, 0])])
def test_orders_match_single_batches(orders, counts):
    Q, gaunt, opts = 20, 1, cb.make_options(tol=1e-6)
    dev = torch.device("cuda", 0)
    u, a0 = [], []
    for k, (order, count) in enumerate(zip(orders, counts)):
        ang = cb.Angular(order, Q, gaunt)
        rows = max(count, 1)
        u.append(cb.sample_moment_vectors(ang, rows, seed=k, s_range=(0.1, 2.0))[0])
        a0.append(cb.isotropic_alpha(ang.n, rows))
    du, da = [torch.from_numpy(x.copy()).to(dev) for x in u], [torch.from_numpy(x.copy()).to(dev) for x in a0]
    it = [torch.full((len(x),), -3, dtype=torch.int32, device=dev) for x in u]
    m = cb.MultiSolver(orders, Q, gaunt, opts)
    torch.cuda.synchronize()
    m.solve_device(counts, du, da, it)
    torch.cuda.synchronize()
    for k, (order, count) in enumerate(zip(orders, counts)):
        gu, ga, gi = du[k].cpu().numpy(), da[k].cpu().numpy(), it[k].cpu().numpy()
        if count == 0:
            assert np.array_equal(gu, u[k]) and np.array_equal(ga, a0[k]) and (gi == -3).all()
            continue
        ctx = cb.Context.for_batches(cb.Angular(order, Q, gaunt), opts)
        ur, ar = u[k].copy(), a0[k].copy()
        its, _, st = ctx.solve_batch(ur, ar)
        ctx.close()
        assert (st == 0).all()
        assert np.array_equal(gu, ur) and np.array_equal(ga, ar) and np.array_equal(gi, its)
    m.close()
