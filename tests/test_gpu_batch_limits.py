"""Boxes where the device, or the part of it that the context may use, holds only
smaller clusters than a box would take, or none: each is solved by the largest
that there is, or by one block, to the bar of the boxes' own test."""
import numpy as np
import pytest

import dare_b200 as D
from tests.helpers import rel_l2
from tests.test_gpu_batched import _oracle_solve
from tests.test_gpu_boxes import _instance

pytestmark = pytest.mark.gpu

SIZES = [(5, 3, 4), (13, 17, 11), (31, 32, 33), (3, 61, 37), (40, 41, 43), (64, 64, 64)]


def test_smaller_clusters():
    ctx = D.Context(0)
    inst = [_instance(n, 3 + q) for q, n in enumerate(SIZES)]
    rng = np.random.default_rng(5)
    fields = [rng.random(int(np.prod(n))) for n in SIZES]
    want = [_oracle_solve(ins, f, 1e-11) for ins, f in zip(inst, fields)]
    solver = D.BiCGStab2({"Convergence Tolerance": 1e-11, "Maximum Iterations": 500, "tol_relative": 1})

    def check(bt, limit):
        for q, f in enumerate(fields):
            bt.set_field(q, f)
        reps = bt.solve(solver)
        xs = [bt.get_field(q) for q in range(len(inst))]
        for q in range(len(inst)):
            assert reps[q]["converged"], (limit, SIZES[q], reps[q])
            assert rel_l2(xs[q], want[q][0]) < 1.3e-10, (limit, SIZES[q])
            assert abs(reps[q]["iters"] - want[q][1]["iters"]) <= 2, (limit, SIZES[q])
        return xs

    kept = D.Batch(ctx, inst)                  # made with every size, limited later
    usual = check(kept, None)
    for limit in (8, 4, 2, 1, 0):
        ctx.set_team_blocks(cluster=limit)
        made = check(D.Batch(ctx, inst), limit)   # made with the limit
        for a, b in zip(made, check(kept, limit)):
            assert np.array_equal(a, b), limit
    ctx.set_team_blocks()
    for a, b in zip(usual, check(kept, None)):
        assert np.array_equal(a, b)
    ctx.set_team_blocks(cluster=2)
    kept.autotune(solver)
    check(kept, "tuned")
