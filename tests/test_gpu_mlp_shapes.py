"""The backward pass at ragged shapes: rows and widths that are no multiple of
its 128- and 64-wide tiles or of 8, one row, one tile more than whole, widths
below and above a tile, n from 3 to 28.  Loss and gradients against the FP64
restatement with BF16 operands, at the bounds of the square case (1e-3 and
2e-2: BF16 rounds at 2^-9, and FP32 sums may round an operand the other way).
"""
import numpy as np
import pytest

import closures_b200 as cb
from test_gpu_mlp import reference_loss_grads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,width,rows", [(1, 8, 64), (2, 40, 37), (2, 20, 129), (3, 64, 1), (4, 72, 128),
                                              (5, 264, 513), (6, 136, 300)])
def test_ragged_gradients(order, width, rows):
    a = cb.Angular(order, 2 * order + 8, 0)
    u, alpha = cb.sample_moment_vectors(a, rows, seed=order, s_range=(0.1, 2.0))
    m = cb.MLP(a.n, width, seed=3)
    mean = np.array([-4.5] + [0.0] * (a.n - 1), np.float32)
    std = np.array([1.5] + [2.0] * (a.n - 1), np.float32)
    m.set_output_scaling(mean, std)
    loss, gW, gb = m.loss_and_grads(u, alpha)
    W, b = m.get_params()
    rloss, rW, rb = reference_loss_grads([w.astype(np.float64) for w in W], [x.astype(np.float64) for x in b], u,
                                         alpha, mean.astype(np.float64), std.astype(np.float64))
    assert abs(loss - rloss) <= 1e-3 * rloss
    for l in range(4):
        assert np.linalg.norm(gW[l] - rW[l]) <= 2e-2 * np.linalg.norm(rW[l]), l
        assert np.linalg.norm(gb[l] - rb[l]) <= 2e-2 * np.linalg.norm(rb[l]), l
    m.close()
