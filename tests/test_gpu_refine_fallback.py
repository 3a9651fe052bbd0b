"""A refinement that is allowed no residual pass at all (max_refinements < 0)
falls back to the FP64 solve with the caller's tolerance, relative or not."""
import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_parity import _hetero_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("relative", [1, 0])
@pytest.mark.parametrize("limit", [-1, 0])
def test_no_refinement_allowed(limit, relative):
    ctx = D.Context(0)
    _, g, f, s, asm, keep = _hetero_system(ctx, 16, seed=2)
    bnorm = float(np.linalg.norm(s.coefficients()[1]))
    tol = 1e-10 if relative else 1e-10 * bnorm
    rep = D.BiCGStab2({"Convergence Tolerance": tol, "Maximum Iterations": 500, "tol_relative": relative,
                       "max_refinements": limit}, precision="FP32_REFINE").solve(s)
    assert rep["converged"] and rep["fallback_used"] == 1 and rep["refinements"] == 0, rep
    assert abs(rep["b_norm"] - bnorm) <= 1e-13 * bnorm
    assert abs(rep["tol_abs"] - 1e-10 * bnorm) <= 1e-13 * 1e-10 * bnorm
    assert rep["true_res_abs"] <= 1.1e-10 * bnorm
