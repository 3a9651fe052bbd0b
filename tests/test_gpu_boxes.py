"""Boxes of a batch solved by clusters of thread blocks (k_boxes in
dare_batched.cu) against the oracle's own assemble + BiCGStab2, at the sizes
where a box is cut: one cell plane to a block and less, remainders in the last
block of a cluster, prime sides, every cluster size, and a box that is too large
for a cluster's shared memory; alone and together, and solved again.

Bar: with V/dt on the diagonal the inverse is bounded by dt/V and the matrix by
kappa V/dt, kappa = 1 + 4 sum_d D dt / dx_d^2 (rows and columns with the
doubled Dirichlet faces included), so a residual of tol ||b|| leaves at most
kappa tol of the solution, from each side.  D dt = 1e-4 and dx >= 1/66 give
kappa < 6.3; tol = 1e-11, the bar 2 * 6.3e-11 = 1.3e-10."""
import numpy as np
import pytest

import dare_b200 as D
from tests.helpers import rel_l2
from tests.test_gpu_batched import _oracle_solve

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (5, 3, 4), (9, 8, 8), (13, 17, 11), (16, 16, 17), (19, 23, 29), (31, 32, 33), (3, 61, 37), (47, 5, 53),
         (40, 41, 43), (50, 49, 48), (64, 64, 64), (66, 65, 64)]


def _instance(n, seed):
    rng = np.random.default_rng(seed)
    bc = {f: (2, 0.0) for f in range(1, 7)}
    bc[1 + seed % 6] = (1, float(rng.uniform(0.0, 1.0)))
    return {"n": n, "size": (1.0, 1.0, 1.0), "D": 1e-2, "dt": 1e-2, "bc": bc}


def _check(ctx, sizes, seed):
    inst = [_instance(n, seed + q) for q, n in enumerate(sizes)]
    rng = np.random.default_rng(seed)
    fields = [rng.random(int(np.prod(n))) for n in sizes]
    bt = D.Batch(ctx, inst)
    solver = D.BiCGStab2({"Convergence Tolerance": 1e-11, "Maximum Iterations": 500, "tol_relative": 1})
    want = [_oracle_solve(ins, f, 1e-11) for ins, f in zip(inst, fields)]
    first = []
    for again in range(2):
        for q, f in enumerate(fields):
            bt.set_field(q, f)
        reps = bt.solve(solver)
        for q in range(len(inst)):
            x = bt.get_field(q)
            assert reps[q]["converged"], (sizes[q], reps[q])
            assert rel_l2(x, want[q][0]) < 1.3e-10, sizes[q]
            assert abs(reps[q]["iters"] - want[q][1]["iters"]) <= 2, sizes[q]
            if again:
                assert np.array_equal(x, first[q]), sizes[q]
            else:
                first.append(x.copy())


@pytest.mark.parametrize("n", SIZES)
def test_one_box(n):
    _check(D.Context(0), [n], sum(n))


def test_boxes_together():
    _check(D.Context(0), SIZES[:-2] + SIZES[:5], 7)
