"""The marching kernels' ring of staged planes at the sizes where it is cut
short: three (the smallest grid) to six planes in all, fewer than or as many as
its stages, odd rows (per-cell copies) and even ones (16-byte copies), bounded and periodic,
FP64 and the FP32-inner refinement, on systems too large for one launch.

The solve stops at 1e-11 of ||b||; the residual recomputed here from the
coefficients may add the rounding of one product (below 1e-13), so the bar is
1.1e-11."""
import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_resident import _apply, _system

pytestmark = pytest.mark.gpu

CASES = [((3, 460, 452), (0, 0, 1)), ((3, 449, 451), (1, 0, 1)), ((4, 397, 401), (1, 1, 0)),
         ((5, 360, 356), (0, 1, 1)), ((6, 330, 332), (1, 0, 0))]


@pytest.mark.parametrize("precision", ["FP64", "FP32_REFINE"])
@pytest.mark.parametrize("n,periodic", CASES)
def test_short_runs(n, periodic, precision):
    ctx = D.Context(0)
    s = D.MatrixSystem(D.Grid(ctx, n, None, 2, periodic))
    diag, rhs, x0 = _system(n, periodic, sum(n))
    s.set_coefficients(diag.reshape(7, -1), rhs.reshape(-1), x0.reshape(-1))
    rep = D.BiCGStab2({"Convergence Tolerance": 1e-11, "Maximum Iterations": 500, "tol_relative": 1},
                      precision=precision).solve(s)
    assert rep["converged"] and not rep["fallback_used"], rep
    x = s.solution().reshape(rhs.shape)
    res = np.linalg.norm(rhs - _apply(diag, x, n, periodic)) / np.linalg.norm(rhs)
    assert res < 1.1e-11
