"""The linear solver's orders 7 to 9 on both sides of the line between a warp per
cell (up to 48 cells per moment) and the parity structure: equal to the oracle
at 1e-12 of the largest density after three steps, the bound of the other
orders, and the host-state step equal to the step to the bit.
"""
import numpy as np
import pytest

import closures_b200 as cb
import decks
import helpers
import pyoracle as oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,nx,ny,filt,ic", [
    (7, 36, 48, "none", "gaussian"), (7, 35, 50, "hauck", "smooth"), (7, 3, 577, "none", "lattice"),
    (8, 40, 54, "sspline", "smooth"), (8, 47, 46, "none", "gaussian"),
    (9, 48, 55, "hauck", "lattice"), (9, 51, 52, "none", "smooth")])
def test_both_sides_of_the_line(tmp_path, order, nx, ny, filt, ic):
    helpers.build_oracle()
    kw = dict(num_cells_x=nx, num_cells_y=ny, init_cond=ic, moment_order=order, quad_order=2 * order + 4,
              filter_type=filt)
    if ic == "lattice":
        kw.update(a_x=-3.5, b_x=3.5, a_y=-3.5, b_y=3.5, floor=1e-10)
    elif ic == "smooth":
        kw.update(a_x=0.0, b_x=1.0, a_y=0.0, b_y=1.0)
    deck = str(tmp_path / "input.deck")
    decks.write_deck(deck, decks.moment_deck_text(**kw))
    o = oracle_lib.GridSolver(deck)
    g, h = cb.Solver(deck, str(tmp_path)), cb.Solver(deck, str(tmp_path))
    host = h.moments().reshape(-1, h.n).copy()
    for _ in range(3):
        o.steps(1)
        g.update(g.max_dt)
        h.step_host(h.max_dt, host)
    mo, mg = o.state()[0][2:-2, 2:-2], g.moments()[2:-2, 2:-2]
    assert np.max(np.abs(mg - mo)) < 1e-12 * np.max(np.abs(mo[:, :, 0]))
    assert np.array_equal(host.reshape(g.moments().shape)[2:-2, 2:-2], mg)
    o.close()
    g.close()
    h.close()
