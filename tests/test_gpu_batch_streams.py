"""The cluster sizes of a batch run side by side on streams that belong to the
context: making a batch costs its allocations (a field of six levels makes about
as many; with streams and events of its own a batch took 1.7 times that), the
batches of a context share them, and handles may go in any order."""
import gc
import time

import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_boxes import _instance

pytestmark = pytest.mark.gpu

SIZES = [(5, 3, 4), (13, 17, 11), (31, 32, 33), (40, 41, 43), (66, 65, 64)]   # several cluster sizes, one block


def _cheapest(make, runs=40):
    best = 1e9
    for _ in range(runs):
        t = time.perf_counter()
        h = make()
        del h
        best = min(best, time.perf_counter() - t)
    return best


def test_making_a_batch_makes_no_streams():
    ctx = D.Context(0)
    g = D.Grid(ctx, (8, 8, 8), None, 2, (0, 0, 0))
    inst = [_instance((8, 8, 8), 1)]
    field = _cheapest(lambda: D.Field(g, 6))
    assert _cheapest(lambda: D.Batch(ctx, inst)) < 1.4 * field


def test_batches_of_a_context_in_any_order():
    solver = D.BiCGStab2({"Convergence Tolerance": 1e-11, "Maximum Iterations": 500, "tol_relative": 1})
    rng = np.random.default_rng(2)
    fields = [rng.random(int(np.prod(n))) for n in SIZES]

    def solve(bt, reports=True):
        for q, f in enumerate(fields):
            bt.set_field(q, f)
        bt.solve(solver, reports=reports)

    result = lambda bt: [bt.get_field(q) for q in range(len(SIZES))]
    ctx = D.Context(0)
    a, b = (D.Batch(ctx, [_instance(n, 9 + q) for q, n in enumerate(SIZES)]) for _ in range(2))
    solve(a)
    want = result(a)
    solve(a, reports=False)      # both in flight
    solve(b, reports=False)
    for x, y, w in zip(result(a), result(b), want):
        assert np.array_equal(x, w) and np.array_equal(y, w)
    solve(b, reports=False)
    del b
    gc.collect()
    solve(a, reports=False)
    for x, w in zip(result(a), want):
        assert np.array_equal(x, w)
    ctx.close()                  # the context before its batch
    del a
    gc.collect()


def test_a_network_shares_them():
    """A minibatch's lanes use the same streams: queued behind a batch that is still
    being solved, replayed from its graph, and after the batch is gone."""
    from tests.test_gpu_unet import _weights
    from tests.test_gpu_unet_training import _pairs
    solver = D.BiCGStab2({"Convergence Tolerance": 1e-11, "Maximum Iterations": 500, "tol_relative": 1})
    rng = np.random.default_rng(4)
    fields = [rng.random(int(np.prod(n))) for n in SIZES]
    ctx = D.Context(0)
    n, count = (16, 24, 32), 4
    r, e = _pairs(n, count, 8)

    def network(c):
        net = D.LearnedPreconditioner(c, n, seed=1)
        net.set_weights(_weights(2, net.num_params))
        return net

    grad = lambda net: net.loss_grad(r.data_ptr(), e.data_ptr(), count)[1]
    want_grad = grad(network(D.Context(0)))
    bt = D.Batch(ctx, [_instance(m, 9 + q) for q, m in enumerate(SIZES)])
    net = network(ctx)
    first = None
    for turn in range(4):
        for q, f in enumerate(fields):
            bt.set_field(q, f)
        bt.solve(solver, reports=False)
        np.testing.assert_array_equal(grad(net), want_grad)
        xs = [bt.get_field(q) for q in range(len(SIZES))]
        first = first or xs
        for x, w in zip(xs, first):
            assert np.array_equal(x, w)
    del bt
    gc.collect()
    np.testing.assert_array_equal(grad(net), want_grad)
