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
