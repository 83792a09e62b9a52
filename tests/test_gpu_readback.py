"""The state comes back as it was set, to the bit, whichever way it is copied.

Copies of 32 MiB and more into pageable memory are shared out to several
threads in 256 KiB chunks (host/readback.cpp).  Sizes: one cell below and one
cell above that limit, a ragged last chunk, whole chunks, a destination at an
odd offset, page-locked memory, and two threads at once.
"""
import threading

import numpy as np
import pytest
import torch

import closures_b200 as cb

pytestmark = pytest.mark.gpu
LIMIT = 32 << 20


def context(NX, NY, seed):
    a = cb.Angular(1, 8, 1)
    C = NX * NY
    rng = np.random.default_rng(seed)
    m, al = rng.normal(size=(C, 3)), rng.normal(size=(C, 3))
    g = cb.cl_grid(NX - 4, NY - 4, 2, 0, 0.0, 0.0, 2.0)
    return cb.Context(g, cb.make_options(), a, np.ones(C), np.ones(C), m, al), m, al


# 24 bytes a cell: 1398101 cells are the last below the limit
@pytest.mark.parametrize("NX,NY", [(9, 7), (1398101 // 811, 811), (5, 279621), (2048, 1024), (1409, 1301)])
def test_state_round_trip(NX, NY):
    ctx, m, al = context(NX, NY, NX)
    for _ in range(2):   # the first call makes the buffers
        gm, ga = ctx.get_state()
        assert np.array_equal(gm.reshape(m.shape), m) and np.array_equal(ga.reshape(al.shape), al)
    ctx.close()


def test_destinations_and_threads():
    ctx, m, al = context(1409, 1301, 1)
    assert m.nbytes > LIMIT
    raw = np.empty(m.size + 1)
    pinned = torch.empty(m.size, dtype=torch.float64, pin_memory=True).numpy()
    for dst in (raw[1:], pinned):
        dst[:] = 0
        assert cb.lib().cl_get_state(ctx._ctx, cb._dp(dst), None) == 0
        assert np.array_equal(dst, m.ravel())
    out = [np.zeros(m.size) for _ in range(4)]
    rc = [1] * 4

    def get(i):
        rc[i] = cb.lib().cl_get_state(ctx._ctx, cb._dp(out[i]), None)

    ts = [threading.Thread(target=get, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert rc == [0] * 4 and all(np.array_equal(o, m.ravel()) for o in out)
    ctx.close()
