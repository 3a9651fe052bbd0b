"""The allocation-free residual norm runs a kernel that a system's solve runs too,
on tiles that need less shared memory (32 x 8 cells instead of 4 x 64): the
system's next solve must not be held to that."""
import numpy as np
import pytest

import dare_b200 as D
from tests.test_zz_no_alloc import _noalloc_norm

pytestmark = pytest.mark.gpu


def _system(ctx, n):
    rng = np.random.default_rng(sum(n))
    g = D.Grid(ctx, n, None, 2, (0, 0, 0))
    s = D.MatrixSystem(g)
    diag = rng.uniform(-1.0, 0.2, size=(7, g.num_cells))
    diag[0] = 1.2 + np.abs(diag[1:]).sum(axis=0)
    s.set_coefficients(diag, rng.normal(size=g.num_cells), np.zeros(g.num_cells))
    return g, s


def test_small_tiles_between_solves():
    import torch
    ctx = D.Context(0)
    torch.cuda.set_device(0)
    stream = torch.cuda.current_stream().cuda_stream
    solver = D.BiCGStab2({"Convergence Tolerance": 1e-10, "Maximum Iterations": 200, "tol_relative": 1})
    _, large = _system(ctx, (600, 400, 3))       # beyond the one-launch solve, rows of three cells
    g, small = _system(ctx, (4, 9, 33))
    zero = np.zeros(large.rows)
    want = solver.solve(large)
    assert want["converged"]
    solver.solve(small)
    out = torch.zeros(1, dtype=torch.float64, device="cuda:0")
    for _ in range(2):
        rc, msg = _noalloc_norm(g, small, out, stream)
        assert rc == 0, msg
        torch.cuda.synchronize()
        large.set_initial_guess(zero)
        assert solver.solve(large) == want
