"""Two networks of one process, whose weight-gradient kernels need different
amounts of shared memory (rows of 200 cells need more than the 48 KB that any
kernel may use, rows of 16 less), train in turn: the order does not matter."""
import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_unet import _weights
from tests.test_gpu_unet_training import _pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(1, 1, 1), (1, 2, 3), (2, 2, 2)])
def test_wide_and_narrow_in_turn(counts):
    ctx = D.Context(0)
    nets = {}
    for n in ((8, 8, 200), (8, 8, 16)):
        net = D.LearnedPreconditioner(ctx, n, seed=1)
        net.set_weights(_weights(3, net.num_params))
        nets[n] = net
    first = {}
    for count in counts:
        for n, net in nets.items():
            r, e = _pairs(n, count, 5)
            grad = net.loss_grad(r.data_ptr(), e.data_ptr(), count)[1]
            assert np.isfinite(grad).all() and np.abs(grad).max() > 0.0
            key = (n, count)
            if key in first:
                np.testing.assert_array_equal(grad, first[key])
            first.setdefault(key, grad)
