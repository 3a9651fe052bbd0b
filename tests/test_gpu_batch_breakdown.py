"""Boxes whose solve breaks down, by one block, by clusters and beside boxes that
converge.  Without diffusion the operator scaled by D^-1 is the identity, and
with small whole numbers for the field every product and sum is exact: alpha =
1, r - alpha v = 0, and the reference leaves its loop at step (14) with step
(10)'s x = x0 + alpha u (BiCGStab2.inl:373-392).  With V = 1 and V / dt = 2 that
is the field itself.  An empty box (field 0, no flux) has rho = 0 at step (4)."""
import numpy as np
import pytest

import dare_b200 as D

pytestmark = pytest.mark.gpu

NEUMANN = {f: (2, 0.0) for f in range(1, 7)}


def _solve(sizes, fields, Ds):
    ctx = D.Context(0)
    inst = [{"n": n, "size": tuple(float(v) for v in n), "D": d, "dt": 0.5, "bc": NEUMANN} for n, d in zip(sizes, Ds)]
    bt = D.Batch(ctx, inst)
    for q, f in enumerate(fields):
        bt.set_field(q, f)
    reps = bt.solve(D.BiCGStab2({"Convergence Tolerance": 1e-12, "Maximum Iterations": 200, "tol_relative": 1}))
    return [bt.get_field(q) for q in range(len(sizes))], reps


@pytest.mark.parametrize("n", [(3, 3, 3), (8, 7, 9), (24, 25, 26), (40, 41, 39), (64, 64, 64), (67, 66, 65)])
def test_breakdown_keeps_step_10(n):
    rng = np.random.default_rng(sum(n))
    f = rng.integers(-3, 4, size=int(np.prod(n))).astype(np.float64)
    (x,), (rep,) = _solve([n], [f], [0.0])
    assert rep["status"] == "breakdown" and rep["breakdown_step"] == 14 and not rep["converged"], rep
    np.testing.assert_array_equal(x, f)


def test_breakdowns_beside_others():
    sizes = [(12, 11, 10), (33, 32, 31), (12, 11, 10), (33, 32, 31), (9, 9, 9), (20, 21, 22)]
    rng = np.random.default_rng(1)
    fields = [rng.integers(-3, 4, size=int(np.prod(n))).astype(np.float64) for n in sizes]
    fields[4][:] = 0.0
    xs, reps = _solve(sizes, fields, [0.0, 0.0, 0.25, 0.25, 0.25, 0.0])
    for q, r in enumerate(reps):
        if q in (0, 1, 5):
            assert r["breakdown_step"] == 14, (q, r)
            np.testing.assert_array_equal(xs[q], fields[q])
        elif q == 4:
            assert r["status"] == "breakdown" and r["breakdown_step"] == 4, r
            assert not xs[q].any()
        else:
            # no flux and an implicit step: the sum is kept
            assert r["converged"] and abs(xs[q].sum() - fields[q].sum()) < 1e-9 * np.abs(fields[q]).sum(), (q, r)
