"""A minibatch on lanes in which a wait of a convolution runs out (a plane that is
never staged, as in the network's own test) reports the time-out once every
lane has ended, and the next call gives the first one's bits."""
import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_unet import _weights
from tests.test_gpu_unet_training import _pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [2, 4])
def test_wait_runs_out_in_a_minibatch(count):
    ctx = D.Context(0)
    n = (16, 24, 32)
    net = D.LearnedPreconditioner(ctx, n, seed=3)
    net.set_weights(_weights(15, net.num_params))
    r, e = _pairs(n, count, 9)
    first = net.loss_grad(r.data_ptr(), e.data_ptr(), count)[1]
    net.set_wait_limit(1000)
    net.debug_skip_plane()
    with pytest.raises(D.DareError) as err:
        net.loss_grad(r.data_ptr(), e.data_ptr(), count)
    assert "timed out" in str(err.value) and "status -6" in str(err.value)
    net.set_wait_limit(0)
    for _ in range(3):
        np.testing.assert_array_equal(net.loss_grad(r.data_ptr(), e.data_ptr(), count)[1], first)
