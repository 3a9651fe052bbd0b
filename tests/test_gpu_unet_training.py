"""The training step's own pieces at the sizes where they are cut: the weight
gradient of the one-channel layers over segments of 1024 padded positions
(planes a little shorter and longer than one segment), and minibatches whose pairs run side by
side on one to four lanes, in turns when there are more pairs than lanes, and
replayed as a graph from the second call on."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import rel_l2
from tests.test_gpu_unet import GRAD_TOL, _torch, _weights

pytestmark = pytest.mark.gpu


def _pairs(n, count, seed):
    torch = _torch()
    g = torch.Generator().manual_seed(seed)
    N = int(np.prod(n))
    r = torch.randn(count, N, generator=g, dtype=torch.float32)
    return r.cuda(), (0.6 * r + 0.4 * torch.randn(count, N, generator=g, dtype=torch.float32)).cuda()


# padded planes of 18 x 58 = 1044, 34 x 34 = 1156, 10 x 98 = 980 and 26 x 42 = 1092 positions
@pytest.mark.parametrize("n", [(8, 16, 56), (16, 32, 32), (8, 8, 96), (24, 24, 40)])
def test_gradient_segments(n):
    import dare_b200 as D
    ctx = D.Context(0)
    net = D.LearnedPreconditioner(ctx, n, seed=1)
    w = _weights(3, net.num_params)
    net.set_weights(w)
    r, e = _pairs(n, 1, 7)
    loss, grad = net.loss_grad(r.data_ptr(), e.data_ptr(), 1)
    oloss, ograd = O.unet_loss_grad(n, w, r.cpu().double().numpy(), e.cpu().double().numpy(), bf16=True)
    assert abs(loss - oloss) < GRAD_TOL * abs(oloss)
    for name, (sl, _) in O.unet_layer_slices().items():
        assert rel_l2(grad[sl], ograd[sl]) < GRAD_TOL, name


@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 9])
def test_minibatch_on_lanes(count):
    """Against the oracle's minibatch gradient at the suite's bar (a pair lost or
    counted twice is off by 1 / count); the replays give the first call's
    bits, and other inputs at other addresses give their own gradient."""
    import dare_b200 as D
    ctx = D.Context(0)
    n = (16, 8, 24)
    net = D.LearnedPreconditioner(ctx, n, seed=1)
    w = _weights(5, net.num_params)
    net.set_weights(w)

    def check(r, e, grad):
        _, ref = O.unet_loss_grad(n, w, r.cpu().double().numpy(), e.cpu().double().numpy(), bf16=True)
        for name, (sl, _) in O.unet_layer_slices().items():
            assert rel_l2(grad[sl], ref[sl]) < GRAD_TOL, name

    r, e = _pairs(n, count, 11)
    first = net.loss_grad(r.data_ptr(), e.data_ptr(), count)[1]
    check(r, e, first)
    for call in range(3):
        np.testing.assert_array_equal(net.loss_grad(r.data_ptr(), e.data_ptr(), count)[1], first)
    r2, e2 = _pairs(n, count, 12)
    check(r2, e2, net.loss_grad(r2.data_ptr(), e2.data_ptr(), count)[1])
