"""Kernel instances shared by solvers of different sizes: a solver created later,
of a lower order or with the other table, must not take away the shared memory
that an earlier one launches with.  Every case interleaves two sizes of one
instance and repeats the earlier result to the bit.
"""
import numpy as np
import pytest
import torch

import closures_b200 as cb
import decks

pytestmark = pytest.mark.gpu


def _vectors(orders, Q, gaunt, count=70):
    dev = torch.device("cuda", 0)
    angs = [cb.Angular(o, Q, gaunt) for o in orders]
    u = [cb.sample_moment_vectors(a, count, seed=k, s_range=(0.1, 1.0))[0] for k, a in enumerate(angs)]
    return angs, u, dev


def _solve(m, u, starts, dev):
    du, da = [torch.from_numpy(x.copy()).to(dev) for x in u], [torch.from_numpy(x.copy()).to(dev) for x in starts]
    torch.cuda.synchronize()
    m.solve_device([len(x) for x in u], du, da)
    torch.cuda.synchronize()
    return [x.cpu().numpy() for x in du + da]


def test_mixed_orders_after_a_direct_table():
    """Orders 1 and 2: one instance for the Gaunt table (staged) and for none."""
    angs, u, dev = _vectors([1, 2], 20, 1)
    a0 = [cb.isotropic_alpha(a.n, len(x)) for a, x in zip(angs, u)]
    m = cb.MultiSolver([1, 2], 20, 1, cb.make_options(tol=1e-6))
    before = _solve(m, u, a0, dev)
    later = [cb.Context.for_batches(cb.Angular(o, 20, 0), cb.make_options(tol=1e-6)) for o in (1, 2)]
    for x, y in zip(before, _solve(m, u, a0, dev)):
        assert np.array_equal(x, y)
    for c in later:
        c.close()
    m.close()


@pytest.mark.parametrize("orders", [[5, 4], [4, 5]])
def test_general_contractions_of_two_orders(orders):
    """PPn without the Gaunt table: orders 4 and 5 run one instance."""
    opts = cb.make_options(moment_type=cb.CL_PPN, tol=1e-6)
    angs, u, dev = _vectors(orders, 20, 0)
    a0 = [cb.isotropic_alpha(a.n, len(x), moment_type=cb.CL_PPN) for a, x in zip(angs, u)]
    m = cb.MultiSolver(orders, 20, 0, opts)
    got = _solve(m, u, a0, dev)
    m.close()
    for k, a in enumerate(angs):
        ctx = cb.Context.for_batches(a, opts)
        ur, ar = u[k].copy(), a0[k].copy()
        _, _, st = ctx.solve_batch(ur, ar)
        ctx.close()
        assert (st == 0).all()
        assert np.array_equal(got[k], ur) and np.array_equal(got[2 + k], ar)


@pytest.mark.parametrize("high,low,gaunt,contraction,cells", [
    (6, 1, 1, "pairs", 20), (6, 1, 1, "single", 20), (3, 1, 0, "pairs", 20), (2, 1, 0, "pairs", 300)])
def test_grid_step_after_a_lower_order(tmp_path, high, low, gaunt, contraction, cells):
    """The flux kernels (whole and shared-out loop) and the screening pass."""
    def solver(order, name):
        deck = str(tmp_path / name)
        decks.write_deck(deck, decks.deck_text(num_cells_x=cells, num_cells_y=cells, gaussian_sigma=0.3, floor=1e-2,
                                               moment_order=order, quad_order=2 * order + 8, tol=1e-6,
                                               use_gaunt=gaunt, extra={"MOMOPT_GPU_CONTRACTION": contraction,
                                                                       "MOMOPT_GPU_TUNE": "0"}))
        return cb.Solver(deck, str(tmp_path))

    first = solver(high, "a.deck")
    first.update(first.max_dt)
    ref = first.context_state()
    first.close()
    s = solver(high, "a.deck")
    other = solver(low, "b.deck")
    s.update(s.max_dt)
    got = s.context_state()
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    other.update(other.max_dt)
    s.close()
    other.close()
