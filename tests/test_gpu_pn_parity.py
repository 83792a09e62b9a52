"""The linear solver's stage on the operators' parity structure, at every order
and at the edges of its tiles: grids of one tile and less, ragged last tiles,
long thin ones, ghost strips wrapped in place (periodic), each filter.

Held to the oracle at 1e-12 of the largest density after three steps, the
bound of the larger grids: a linear step of some 10^2 sums of terms of that
size, 10 to 100 roundings of 1e-16 each.
"""
import numpy as np
import pytest

import closures_b200 as cb
import decks
import helpers
import pyoracle as oracle_lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,nx,ny,filt,ic", [
    (1, 1, 1, "none", "gaussian"), (1, 33, 7, "hauck", "smooth"), (2, 16, 16, "lanczos", "smooth"),
    (2, 3, 65, "none", "lattice"), (3, 17, 15, "sspline", "gaussian"), (3, 8, 5, "none", "smooth"),
    (4, 31, 2, "hauck", "lattice"), (5, 9, 40, "none", "smooth"), (6, 15, 33, "lanczos", "gaussian"),
    (6, 5, 4, "hauck", "smooth"), (7, 12, 19, "none", "gaussian"), (8, 7, 16, "sspline", "smooth"),
    (9, 18, 6, "hauck", "lattice")])
def test_stage_edges(tmp_path, order, nx, ny, filt, ic):
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
    g = cb.Solver(deck, str(tmp_path))
    for _ in range(3):
        o.steps(1)
        g.update(g.max_dt)
    mo, mg = o.state()[0][2:-2, 2:-2], g.moments()[2:-2, 2:-2]
    assert np.max(np.abs(mg - mo)) < 1e-12 * np.max(np.abs(mo[:, :, 0]))
    o.close()
    g.close()
