"""One slab holds the whole grid and is solved as such: its report carries what
the single grid's does, the recomputed residual ||b - A x||_2 among it, and
leaves it out when it is not asked for."""
import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_slabs import SHAPES, Setup, _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", ["JACOBI", "NONE"])
@pytest.mark.parametrize("periodic_x", [1, 0])
@pytest.mark.parametrize("n", SHAPES)
def test_one_slab_reports_the_true_residual(n, periodic_x, precond):
    ctx = D.Context(0)
    st = Setup(ctx, _case(n, periodic_x), 1)
    st.s.build(st.f, st.asm)
    x0 = st.s.solution()
    tol = 1e-11 * float(np.linalg.norm(st.s.coefficients()[1]))
    reports = []
    for asked in (1, 0):
        solver = D.BiCGStab2({"Convergence Tolerance": tol, "Maximum Iterations": 2000, "compute_true_residual": asked},
                             precond=precond)
        st.s.set_initial_guess(x0)
        st.sl.assemble(st.slab_asm)
        whole, slab = solver.solve(st.s), st.sl.solve(solver)
        assert np.array_equal(st.sl.solution(), st.s.solution())
        assert slab == whole
        reports.append(slab)
    assert 0.0 < reports[0]["true_res_abs"] <= 1.1 * tol
    assert reports[1]["true_res_abs"] == 0.0
