"""K1's order of a stage's cells, sorted by several CTAs in blocks of 1024: grids
with ghosts of 1024 cells, one more, one block less and one more than three.
A cell left out would keep its start, one taken twice would be counted twice:
every cell takes an iteration, the solves counted are whole stages, and two RK2
steps match the oracle's moments to 1e-10 relative (the suite's bound where
rounding decides nothing).
"""
import numpy as np
import pytest

import closures_b200 as cb
import decks
import pyoracle as oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NX,NY", [(32, 32), (25, 41), (11, 93), (37, 83)])
@pytest.mark.parametrize("screen", [True, False])
def test_every_cell_once(tmp_path, NX, NY, screen):
    deck = str(tmp_path / "input.deck")
    decks.write_deck(deck, decks.deck_text(num_cells_x=NX - 4, num_cells_y=NY - 4, gaussian_sigma=0.4, floor=1e-2,
                                           moment_order=3, quad_order=10, tol=1e-6, use_gaunt=1, moment_type="mn"))
    s = cb.Solver(deck, str(tmp_path))
    if not screen:
        cb._check(cb.lib().cl_set_range_test(cb.lib().cl_solver_context(s._s), 0), lambda: b"")
    g = oracle_lib.GridSolver(deck)
    for _ in range(2):
        s.update(s.max_dt)
        g.steps(1)
        it = s.last_iterations()
        assert it.min() >= 1
    assert s.stats()["num_solves"] % (NX * NY) == 0
    m_g, m_o = s.context_state()[0], g.state()[0]
    assert np.max(np.abs(m_g - m_o) / np.abs(m_o[:, :, :1])) < 1e-10
    s.close()
    g.close()
