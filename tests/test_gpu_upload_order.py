"""A state set from pageable memory is there before the first kernel that reads
it: repeated uploads of changing states, each followed at once by a step, give
the bits of the first time, in both solvers.
"""
import numpy as np
import pytest

import closures_b200 as cb
import decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,nx,ny", [(8, 40, 54), (3, 120, 90), (6, 90, 70)])
def test_linear_solver(tmp_path, order, nx, ny):
    deck = str(tmp_path / "input.deck")
    decks.write_deck(deck, decks.moment_deck_text(num_cells_x=nx, num_cells_y=ny, init_cond="smooth",
                                                  moment_order=order, quad_order=2 * order + 4, filter_type="none",
                                                  a_x=0.0, b_x=1.0, a_y=0.0, b_y=1.0))
    s = cb.Solver(deck, str(tmp_path))
    rng = np.random.default_rng(order)
    states = [rng.uniform(0.5, 1.5, (s.NX * s.NY, s.n)) for _ in range(3)]
    ref = [None] * 3
    for k in range(60):
        host = states[k % 3].copy()
        s.step_host(s.max_dt, host)
        got = host.reshape(s.NX, s.NY, s.n)[2:-2, 2:-2]
        if ref[k % 3] is None:
            ref[k % 3] = got.copy()
        assert np.array_equal(got, ref[k % 3]), k
    s.close()


def test_momopt_solver(tmp_path):
    deck = str(tmp_path / "input.deck")
    decks.write_deck(deck, decks.deck_text(num_cells_x=150, num_cells_y=110, gaussian_sigma=0.3, floor=1e-2,
                                           moment_order=2, quad_order=12, tol=1e-6,
                                           extra={"MOMOPT_GPU_TUNE": "0"}))
    s = cb.Solver(deck, str(tmp_path))
    ctx = s.context()
    m, a = ctx.get_state()
    states = [(f * m.reshape(-1, s.n), a.reshape(-1, s.n).copy()) for f in (1.0, 1.5, 0.75)]
    ref = [None] * 3
    for k in range(30):
        mk, ak = states[k % 3]
        ctx.set_state(mk, ak)
        s.update(s.max_dt)
        got = ctx.get_state()[0]
        if ref[k % 3] is None:
            ref[k % 3] = got.copy()
        assert np.array_equal(got, ref[k % 3]), k
    s.close()
