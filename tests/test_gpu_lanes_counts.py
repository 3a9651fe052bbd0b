"""Minibatches of different pair counts in turn, as at the end of a pass over the
data: each count's gradient keeps its bits, and no count pays for the launches'
graph again because another one came between.  (Steady calls of 16^3 take
0.4 ms as a graph, 0.9 ms launch by launch and 1.4 ms with a graph built anew.)"""
import time

import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_unet import _weights
from tests.test_gpu_unet_training import _pairs

pytestmark = pytest.mark.gpu

COUNTS = (4, 4, 3, 3, 8, 8)


def test_counts_in_turn():
    ctx = D.Context(0)
    n = (16, 16, 16)
    r, e = _pairs(n, max(COUNTS), 2)

    def network():
        net = D.LearnedPreconditioner(ctx, n, seed=1)
        net.set_weights(_weights(6, net.num_params))
        return net

    def call(net, count):
        t = time.perf_counter()
        grad = net.loss_grad(r.data_ptr(), e.data_ptr(), count)[1]
        return time.perf_counter() - t, grad

    alone = {}
    for count in set(COUNTS):
        net = network()
        grads = [call(net, count) for _ in range(13)]
        for _, g in grads:
            np.testing.assert_array_equal(g, grads[0][1])
        alone[count] = (float(np.median([t for t, _ in grads[3:]])), grads[0][1])
    net = network()
    times = {}
    for turn in range(14):
        for place, count in enumerate(COUNTS):
            t, g = call(net, count)
            np.testing.assert_array_equal(g, alone[count][1])
            if turn > 2:
                times.setdefault((place, count), []).append(t)
    for (place, count), ts in times.items():
        assert np.median(ts) < 1.8 * alone[count][0], (place, count, np.median(ts), alone[count][0])
