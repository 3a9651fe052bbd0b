"""Boxes without diffusion, whose scaled operator A D^-1 is the identity: the own
value of a row is the operand itself, unrounded, whatever the centre coefficient
is (here 1 / 0.3 and the like, so that scaling by its inverse and back would round).
Then v = r bit for bit, the two dot products of alpha add the same numbers in the
same way (five boxes a size: one rounding that differs shows in a few of a hundred), alpha
= 1, r - alpha v = 0, and the solve ends as the reference's does, in step (14)
with step (10)'s x = x0 + alpha u: M^-1 (x0 + (b - x0)) = M^-1 b, the field
itself up to the rounding of x0 + (b - x0) and of the two scalings (8 units
roundoff of the largest of x0, b and their sum, |b| = tt |x0|, over tt)."""
import numpy as np
import pytest

import dare_b200 as D

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (7, 5, 6), (12, 12, 12), (16, 16, 16), (24, 20, 22), (31, 32, 33), (40, 41, 43)] * 5 + [(67, 66, 65)]


@pytest.mark.parametrize("tol", [1e-10, 0.0])
@pytest.mark.parametrize("dt", [0.3, 0.7, 3.0])
def test_identity(dt, tol):
    ctx = D.Context(0)
    rng = np.random.default_rng(3)
    inst = [{"n": n, "size": tuple(1.1 * v for v in n), "D": 0.0, "dt": dt, "bc": {f: (2, 0.0) for f in range(1, 7)}}
            for n in SIZES]
    bt = D.Batch(ctx, inst)
    fields = [rng.normal(size=int(np.prod(n))) for n in SIZES]
    for q, f in enumerate(fields):
        bt.set_field(q, f)
    reps = bt.solve(D.BiCGStab2({"Convergence Tolerance": tol, "Maximum Iterations": 100, "tol_relative": 1}))
    tt = 1.1 ** 3 / dt
    bar = 8 * 2.0 ** -53 * (2 + max(tt, 1.0)) / tt
    for q, (f, rep) in enumerate(zip(fields, reps)):
        assert rep["status"] == "breakdown" and rep["breakdown_step"] == 14 and rep["iters"] == 1, (SIZES[q], rep)
        assert np.abs(bt.get_field(q) - f).max() <= bar * np.abs(f).max(), SIZES[q]
