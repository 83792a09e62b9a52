"""Periodic grids of one and two cells a side, where ghost strips wrap onto each
other: both solvers against the oracle, and the ghosts that a step leaves in
the linear solver's second buffer.

Linear steps are held to 1e-12 of the largest density (some 10^2 sums of terms
of that size), momopt steps to the suite's 1e-10 per cell.
"""
import ctypes as C

import numpy as np
import pytest

import closures_b200 as cb
import decks
import helpers
import pyoracle as oracle_lib

pytestmark = pytest.mark.gpu

SIZES = [(1, 7), (6, 1), (1, 1), (2, 2), (2, 1), (1, 2), (3, 2)]


def _varied(shape, n, seed):
    """A state that differs from cell to cell (the decks' own is close to
    uniform on so few cells): u_0 in 1..2, the others small against it."""
    rng = np.random.default_rng(seed)
    m = 0.1 * rng.uniform(-1.0, 1.0, shape + (n,))
    m[:, :, 0] = rng.uniform(1.0, 2.0, shape)
    return m


@pytest.mark.parametrize("order", [1, 3, 6])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_linear_steps(tmp_path, nx, ny, order):
    helpers.build_oracle()
    deck = str(tmp_path / "input.deck")
    decks.write_deck(deck, decks.moment_deck_text(num_cells_x=nx, num_cells_y=ny, init_cond="smooth",
                                                  moment_order=order, quad_order=2 * order + 4, filter_type="none",
                                                  a_x=0.0, b_x=1.0, a_y=0.0, b_y=1.0))
    o = oracle_lib.GridSolver(deck)
    g = cb.Solver(deck, str(tmp_path))
    m0 = _varied((nx + 4, ny + 4), g.n, order)
    o.set_state(m0, np.zeros_like(m0))
    g.set_moments(m0)
    for _ in range(4):
        o.steps(1)
        g.update(g.max_dt)
    mo, mg = o.state()[0][2:-2, 2:-2], g.moments()[2:-2, 2:-2]
    assert np.max(np.abs(mg - mo)) < 1e-12 * np.max(np.abs(m0))
    o.close()
    g.close()


@pytest.mark.parametrize("nx,ny", SIZES)
def test_momopt_steps(tmp_path, nx, ny):
    helpers.build_oracle()
    deck = str(tmp_path / "input.deck")
    decks.write_deck(deck, decks.deck_text(num_cells_x=nx, num_cells_y=ny, init_cond="smooth", moment_order=2,
                                           quad_order=12, tol=1e-8, a_x=0.0, b_x=1.0, a_y=0.0, b_y=1.0))
    o = oracle_lib.GridSolver(deck)
    g = cb.Solver(deck, str(tmp_path))
    _, a0 = o.state()
    m0 = _varied((nx + 4, ny + 4), g.n, 2)
    o.set_state(m0, a0)
    g.context().set_state(m0.reshape(-1, g.n), a0.reshape(-1, g.n))
    for _ in range(3):
        o.steps(1)
        g.update(g.max_dt)
    mo, mg = o.state()[0][2:-2, 2:-2], g.context_state()[0][2:-2, 2:-2]
    assert np.max(np.abs(mg - mo) / np.abs(mo[:, :, :1])) < 1e-10
    o.close()
    g.close()


def test_second_buffer_ghosts(tmp_path):
    """A step leaves the buffer between its stages with the ghosts of its
    second stage: a stage run by itself afterwards shows them."""
    nx, ny = 5, 4
    deck = str(tmp_path / "input.deck")
    decks.write_deck(deck, decks.moment_deck_text(num_cells_x=nx, num_cells_y=ny, init_cond="smooth",
                                                  moment_order=3, quad_order=10, filter_type="none",
                                                  a_x=0.0, b_x=1.0, a_y=0.0, b_y=1.0))
    g = cb.Solver(deck, str(tmp_path))
    L, pn = cb.lib(), C.c_void_p(cb.lib().cl_solver_pn(g._s))
    n, dt = g.n, C.c_double(g.max_dt)
    dx, dy = C.c_double(g.dx), C.c_double(g.dy)

    def wrap(m):
        m = m.copy()
        m[:2, 2:-2], m[-2:, 2:-2] = m[-4:-2, 2:-2], m[2:4, 2:-2]
        m[2:-2, :2], m[2:-2, -2:] = m[2:-2, -4:-2], m[2:-2, 2:4]
        return m

    def state():
        out = np.empty((nx + 4, ny + 4, n))
        assert L.cl_pn_get_state(pn, out.ctypes.data_as(C.POINTER(C.c_double))) == 0
        return out

    m0 = wrap(_varied((nx + 4, ny + 4), n, 9))
    g.set_moments(m0)
    assert L.cl_pn_stage(pn, 1, dt, dx, dy) == 0
    between = wrap(state())          # the first stage's result, as the second stage reads it
    g.set_moments(m0)
    g.update(g.max_dt)
    assert L.cl_pn_stage(pn, 1, dt, dx, dy) == 0
    after = state()
    for strip in (np.s_[:2, 2:-2], np.s_[-2:, 2:-2], np.s_[2:-2, :2], np.s_[2:-2, -2:]):
        assert np.array_equal(after[strip], between[strip])
    g.close()
