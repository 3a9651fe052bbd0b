"""One-launch solves where the device, or the part of it that the context may use,
does not hold the usual team: a smaller cluster, fewer blocks of the device, the
device's blocks in place of a cluster, and the marching kernels in place of
both.  Each solves the system, to the tolerance asked for."""
import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_resident import _apply, _system

pytestmark = pytest.mark.gpu


# (cluster blocks, device blocks) -> one launch?
LIMITS = [(-1, -1, True), (8, -1, True), (1, 0, None), (0, -1, True), (0, 20, True), (3, 3, None), (0, 0, False)]


@pytest.mark.parametrize("precond", ["JACOBI", "NONE"])
@pytest.mark.parametrize("n", [(9, 8, 10), (25, 24, 26), (34, 33, 32)])
def test_fewer_blocks(n, precond):
    periodic = (1, 0, 1)
    ctx = D.Context(0)
    g = D.Grid(ctx, n, None, 2, periodic)
    s = D.MatrixSystem(g)
    diag, rhs, x0 = _system(n, periodic, sum(n))
    solver = D.BiCGStab2({"Convergence Tolerance": 1e-11, "Maximum Iterations": 500, "tol_relative": 1}, precond=precond)
    for cluster, grid, one in LIMITS:
        ctx.set_team_blocks(cluster, grid)
        s.set_coefficients(diag.reshape(7, -1), rhs.reshape(-1), x0.reshape(-1))
        launches = ctx.launch_count
        rep = solver.solve(s)
        launches = ctx.launch_count - launches
        assert rep["converged"], (cluster, grid, rep)
        x = s.solution().reshape(rhs.shape)
        res = np.linalg.norm(rhs - _apply(diag, x, n, periodic)) / np.linalg.norm(rhs)
        assert res < 1.1e-11, (cluster, grid)
        if one is not None:
            assert (launches == 1) == one, (cluster, grid, launches)
    # and the usual team again
    ctx.set_team_blocks()
    launches = ctx.launch_count
    solver.solve(s)
    assert ctx.launch_count - launches == 1
