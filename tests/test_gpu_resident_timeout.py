"""Waits between the blocks of a one-launch solve that run out.  The solve ends,
reports DARE_ERR_TIMEOUT whichever block gave up and whatever the others got, and
the next one on the same system gives the bits of the first."""
import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_resident import _system

pytestmark = pytest.mark.gpu

N = (33, 34, 35)   # 39270 cells: blocks of the whole device, not of one cluster


def _setup(diagonal=False):
    ctx = D.Context(0)
    g = D.Grid(ctx, N, None, 2, (1, 0, 1))
    s = D.MatrixSystem(g)
    diag, rhs, x0 = _system(N, (1, 0, 1), 3)
    if diagonal:
        diag[1:] = 0.0
        diag[0] = 2.0
    s.set_coefficients(diag.reshape(7, -1), rhs.reshape(-1), x0.reshape(-1))
    return ctx, s, rhs.reshape(-1), x0.reshape(-1)


def _solver(precond="JACOBI", **kw):
    return D.BiCGStab2({"Convergence Tolerance": 1e-11, "Maximum Iterations": 500, "tol_relative": 1, **kw},
                       precond=precond)


@pytest.mark.parametrize("precond", ["JACOBI", "NONE"])
def test_waits_run_out(precond):
    ctx, s, _, x0 = _setup()
    solver = _solver(precond)
    want = solver.solve(s)
    x = s.solution()
    assert want["converged"]
    ctx.set_wait_limit(1)
    s.set_initial_guess(x0)
    with pytest.raises(D.DareError) as err:
        solver.solve(s)
    assert "ran out" in str(err.value) and "status -6" in str(err.value)
    ctx.set_wait_limit(0)
    for _ in range(2):
        s.set_initial_guess(x0)
        assert solver.solve(s) == want
        assert np.array_equal(s.solution(), x)


@pytest.mark.parametrize("block", [0, 5, 66])
def test_one_block_gives_up_at_the_last_exchange(block):
    """A = 2 I and x0 = b / 2: without a preconditioner the initial residual's
    exchange is the only one.  The other blocks get its total and finish."""
    ctx, s, rhs, _ = _setup(diagonal=True)
    solver = _solver("NONE", compute_true_residual=0)
    s.set_initial_guess(rhs / 2)
    want = solver.solve(s)
    assert want["converged"] and want["iters"] == 0
    ctx.debug_give_up(block)
    with pytest.raises(D.DareError) as err:
        solver.solve(s)
    assert "ran out" in str(err.value) and "status -6" in str(err.value)
    assert solver.solve(s) == want
    assert np.array_equal(s.solution(), rhs / 2)


def test_one_block_gives_up_first():
    """... at the first exchange of many: the blocks that wait for it give up too."""
    ctx, s, _, x0 = _setup()
    solver = _solver()
    want = solver.solve(s)
    ctx.set_wait_limit(20000)
    ctx.debug_give_up(7)
    s.set_initial_guess(x0)
    with pytest.raises(D.DareError):
        solver.solve(s)
    ctx.set_wait_limit(0)
    s.set_initial_guess(x0)
    assert solver.solve(s) == want
