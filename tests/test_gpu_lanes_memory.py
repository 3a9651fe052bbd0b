"""A minibatch whose pairs could run side by side goes on one after another
where the device has no room for the other pairs' activations, and without the
graph of its launches where it has none for the graph's inputs: the gradient is
the same to the bit (two pairs are added in their order either way), also when
the room comes back."""
import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_unet import _torch, _weights
from tests.test_gpu_unet_training import _pairs

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _fill(torch, leave):
    """Blocks that hold all of the device's memory but `leave` bytes."""
    torch.cuda.empty_cache()
    held = []
    for size in (4096 * MB, 64 * MB, 2 * MB):
        while torch.cuda.mem_get_info()[0] - leave >= size:
            n = (torch.cuda.mem_get_info()[0] - leave) // size
            held.append(torch.empty(n * size, dtype=torch.uint8, device="cuda"))
    return held


# 96^3: the activations of a pair take about 100 MB, the graph's inputs of two
# pairs 14 MB
@pytest.mark.parametrize("leave", [64, 8])
def test_minibatch_without_room(leave):
    torch = _torch()
    ctx = D.Context(0)
    n, count = (96, 96, 96), 2
    r, e = _pairs(n, count, 3)

    def network():
        net = D.LearnedPreconditioner(ctx, n, seed=1)
        net.set_weights(_weights(4, net.num_params))
        return net

    grads = lambda net: net.loss_grad(r.data_ptr(), e.data_ptr(), count)[1]
    net = network()
    want = [grads(net) for _ in range(3)][-1]
    del net
    net = network()
    net.loss_grad(r.data_ptr(), e.data_ptr(), 1)   # what every call needs is there
    held = _fill(torch, leave * MB)
    try:
        got = [grads(net) for _ in range(3)]
    finally:
        del held
        torch.cuda.empty_cache()
    got += [grads(net) for _ in range(3)]
    for g in got:
        np.testing.assert_array_equal(g, want)
