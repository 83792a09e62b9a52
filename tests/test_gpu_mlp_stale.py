"""Gradients of one call do not depend on what an earlier call left in the work
buffers: widths that are no multiple of 8, whose padding columns lie over
another layer's gradients of the call before.  The earlier call has targets
that are not finite in the rows the later one does not use; the later one must
give the bits of a fresh network.
"""
import numpy as np
import pytest

import closures_b200 as cb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,width", [(3, 20), (2, 12), (4, 100), (6, 25), (3, 64)])
def test_gradients_after_a_diverged_call(order, width):
    a = cb.Angular(order, 2 * order + 8, 0)
    u, alpha = cb.sample_moment_vectors(a, 512, seed=order, s_range=(0.1, 2.0))
    bad = alpha.copy()
    bad[100:] = np.nan
    out = []
    for first in (True, False):
        m = cb.MLP(a.n, width, seed=3)
        if first:
            m.loss_and_grads(u, bad)
        out.append(m.loss_and_grads(u[:200], alpha[:200]))
        m.close()
    (l1, gW1, gb1), (l2, gW2, gb2) = out
    assert np.isfinite(l1) and l1 == l2
    for x, y in zip(list(gW1) + list(gb1), list(gW2) + list(gb2)):
        assert np.isfinite(x).all() and np.array_equal(x, y)
