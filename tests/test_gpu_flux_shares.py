"""K2+K3 on grids of few tiles, where the direction loop is shared out over
CTAs and projected by a second kernel: tile edges, remainders and both tile
layouts, one RK2 step against the oracle (1e-10 relative, the suite's bound
where rounding decides nothing; 4 / 25 ... chunks per tile leave uneven shares).
"""
import numpy as np
import pytest

import closures_b200 as cb
import decks
import pyoracle as oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,order,Q,closure,contraction", [
    (1, 1, 1, 4, "mn", "pairs"), (5, 3, 2, 8, "mn", "pairs"), (16, 16, 3, 10, "mn", "pairs"),
    (17, 33, 2, 20, "mn", "single"), (47, 16, 3, 10, "ppn", "pairs"), (33, 17, 2, 8, "ppn", "single")])
def test_small_grid_step(tmp_path, nx, ny, order, Q, closure, contraction):
    deck = str(tmp_path / "input.deck")
    decks.write_deck(deck, decks.deck_text(num_cells_x=nx, num_cells_y=ny, gaussian_sigma=0.4, floor=1e-2,
                                           moment_order=order, quad_order=Q, tol=1e-6, use_gaunt=0,
                                           moment_type=closure, extra={"MOMOPT_GPU_CONTRACTION": contraction}))
    s = cb.Solver(deck, str(tmp_path))
    g = oracle_lib.GridSolver(deck)
    s.update(s.max_dt)
    g.steps(1)
    m_g, _ = s.context_state()
    m_o, _ = g.state()
    assert np.max(np.abs(m_g - m_o) / np.abs(m_o[:, :, :1])) < 1e-10
    assert s.stats()["flux_tiles"] <= 2 * -(-nx // 16) * -(-ny // 16)
    s.close()
    g.close()
