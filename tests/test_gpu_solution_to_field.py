"""The pass that writes a step's solution into the field with its periodic
ghosts (k_solution_to_field in dare_core.cu) against CopyTo and
ExchangeHaloCells one after the other, bit for bit with every ghost: after a
refinement (x as it is) and after a marching FP64 solve (x = M^-1 y), rows
shorter and longer than a block, fewer rows than a block's share and remainders,
one to three dimensions, every kind of periodicity."""
import numpy as np
import pytest

import dare_b200 as D

pytestmark = pytest.mark.gpu

CASES = [((700,), (1,), "FP32_REFINE"), ((300001,), (1,), "FP32_REFINE"), ((37, 1029), (1, 0), "FP32_REFINE"),
         ((1029, 3), (0, 1), "FP32_REFINE"), ((19, 23, 300), (1, 1, 1), "FP32_REFINE"),
         ((5, 300, 7), (0, 1, 1), "FP32_REFINE"), ((41, 3, 11), (1, 0, 1), "FP32_REFINE"),
         ((600001,), (1,), "FP64"), ((767, 803), (1, 1), "FP64"), ((83, 91, 81), (0, 1, 1), "FP64")]


@pytest.mark.parametrize("n,periodic,precision", CASES)
def test_matches_copy_and_exchange(n, periodic, precision):
    ctx = D.Context(0)
    g = D.Grid(ctx, n, (1.0,) * len(n), 2, periodic)
    f, twin, s = D.Field(g, 2), D.Field(g, 2), D.MatrixSystem(g)
    phi = np.random.default_rng(sum(n)).random(g.num_cells_ghosted)
    for field in (f, twin):
        for level in (0, 1):
            field.upload(phi, level)
    h = min(1.0 / v for v in n)
    asm = D.Assembly(dt=1e-2, D=0.2 * h * h / 1e-2)
    solver = D.BiCGStab2({"Convergence Tolerance": 1e-10, "Maximum Iterations": 200, "tol_relative": 1,
                          "compute_true_residual": 0}, precision=precision)
    rep = D.timestep(s, f, asm, solver)
    assert rep["converged"], rep
    s.copy_to(twin)
    twin.exchange_halo()
    np.testing.assert_array_equal(f.download(0), twin.download(0))
