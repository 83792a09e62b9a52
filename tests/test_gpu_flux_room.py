"""The buffer of the shared-out direction loop is reserved only where a launch of
the grid uses it, and a context for batches reserves none.

148 tiles (one wave) at 100 chunks of directions are better left whole; the
buffer would take 148 x 100 x 32 KiB = 463 MiB.  The same chunks on 80 tiles are
shared out.  The state of these grids takes under 4 MiB; device memory comes in
blocks of 2 MiB.
"""
import numpy as np
import pytest
import torch

import closures_b200 as cb

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _context(nx, ny, Q):
    a = cb.Angular(1, Q, 0)
    cells = (nx + 4) * (ny + 4)
    m = np.zeros((cells, a.n))
    m[:, 0] = 1.0
    grid = cb.cl_grid(nx, ny, 2, 0, 0.0, 0.0, 2.0)
    return cb.Context(grid, cb.make_options(), a, np.ones(cells), np.ones(cells), m,
                      cb.isotropic_alpha(a.n, cells))


@pytest.mark.parametrize("nx,ny,reserved", [(64, 592, False), (1, 1, False), (64, 320, True)])
def test_reserved_memory(nx, ny, reserved):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the rule's line depends on the number of SMs")
    warm = _context(nx, ny, 40)   # kernels loaded
    warm.step(1e-3, 0.1, 0.1)
    warm.close()
    free = torch.cuda.mem_get_info()[0]
    ctx = _context(nx, ny, 40)
    used = free - torch.cuda.mem_get_info()[0]
    buffer = 100 * 32 * 1024 * (-(-nx // 16)) * (-(-ny // 16))
    if reserved:
        assert used >= buffer
    elif buffer > 64 * MIB:
        assert used < 64 * MIB
    else:
        assert used < buffer or used <= 2 * MIB
    ctx.step(1e-3, 0.1, 0.1)
    ctx.close()


@pytest.mark.parametrize("nx,ny", [(16 * 5, 16 * 30), (16 * 13 - 3, 16 * 13 - 9), (16 * 8, 16 * 37), (16, 16 * 149)])
@pytest.mark.parametrize("contraction", [cb.CL_CONTRACT_PAIRS, cb.CL_CONTRACT_SINGLE])
def test_more_than_a_wave(nx, ny, contraction):
    """Grids of more than a wave of tiles (150, 169, 296, 149): every tile has the
    result of the same cells of a grid of few tiles, whose shares are others."""
    a = cb.Angular(2, 20, 0)

    def step(x0, y0, cells_x, cells_y):
        # the state of cell (i, j) of the whole grid, ghosts included, from i and j alone
        i, j = np.meshgrid(np.arange(cells_x + 4) + x0, np.arange(cells_y + 4) + y0, indexing="ij")
        m = np.zeros(i.shape + (a.n,))
        m[..., 0] = 1.5 + np.sin(0.37 * i) * np.cos(0.21 * j)
        for k in range(1, a.n):
            m[..., k] = 0.1 * np.sin(0.13 * k * i + 0.29 * j)
        flat = m.reshape(-1, a.n)
        cells = len(flat)
        grid = cb.cl_grid(cells_x, cells_y, 2, 0, 0.0, 0.0, 2.0)
        ctx = cb.Context(grid, cb.make_options(contraction=contraction), a, np.ones(cells), 0.5 * np.ones(cells), flat,
                         cb.isotropic_alpha(a.n, cells))
        ctx.step_timed(1e-2, 0.1, 0.1)
        out = ctx.get_state()[0]
        ctx.close()
        return out

    whole = step(0, 0, nx, ny)
    # a step reaches four cells (two stages of two): the last tile and its
    # neighbourhood, cut out where the cut is farther away than that
    cx, cy = min(nx, 40), min(ny, 40)
    part = step(nx - cx, ny - cy, cx, cy)
    ix, iy = 2 + (8 if cx < nx else 0), 2 + (8 if cy < ny else 0)
    assert np.array_equal(part[ix:-2, iy:-2], whole[nx - cx:][ix:-2, (ny - cy) + iy:-2])
