"""The one-launch solve of small systems (dare_resident.cu) at the sizes where
its blocks are cut: one block, a remainder in the last block, the largest single
cluster and the first cooperative launch, one to four cells a thread, the largest system it takes and the first one that goes to the
marching kernels; every mix of periodic and bounded directions, one to three
dimensions, two components, with and without Jacobi.

The solve stops at 1e-11 of ||b|| by its recurrence; the residual recomputed
here from the coefficients may add the rounding of one product (7 terms, a
unit roundoff each, on vectors of the size of b: below 1e-13), so the bar is
1.1e-11.  Where the oracle's solve is affordable the solution is compared too,
at the suite's 1e-9."""
import numpy as np
import pytest

import dare_b200 as D
from oracle import oracle as O
from tests.helpers import diag_to_csr, rel_l2

pytestmark = pytest.mark.gpu


def _system(n, periodic, seed, comps=1):
    """Random diagonally dominant rows; removed neighbours carry a value that
    must not be used."""
    rng = np.random.default_rng(seed)
    shape = tuple(n) + (1,) * (3 - len(n))
    diag = rng.uniform(-1.0, 0.2, size=(7, comps) + shape)
    for d in range(3):
        if d >= len(n):
            diag[2 * d + 1:2 * d + 3] = 0.0
    diag[0] = 1.2 + np.abs(diag[1:]).sum(axis=0)
    return diag, rng.normal(size=(comps,) + shape), rng.normal(size=(comps,) + shape)


def _apply(diag, x, n, periodic):
    y = diag[0] * x
    for d in range(len(n)):
        for side in range(2):
            v = np.roll(x, 1 - 2 * side, axis=1 + d)
            if not periodic[d]:
                edge = [slice(None)] * 4
                edge[1 + d] = 0 if side == 0 else n[d] - 1
                v[tuple(edge)] = 0.0
            y = y + diag[2 * d + 1 + side] * v
    return y


CASES = [((3, 3, 3), (0, 0, 0), 1), ((8, 8, 8), (1, 1, 1), 1), ((8, 8, 9), (0, 1, 0), 1), ((17, 13, 10), (1, 0, 1), 1),
         ((5, 700), (0, 1), 1), ((3000,), (1,), 1), ((4000,), (0,), 2), ((40, 33), (1, 0), 2), ((12, 11, 9), (0, 0, 1), 2),
         ((32, 32, 32), (1, 0, 1), 1), ((33, 32, 32), (0, 1, 1), 1), ((53, 54, 52), (1, 1, 0), 1), ((66, 65, 67), (0, 1, 1), 1), ((76, 75, 77), (1, 0, 1), 1),
         ((83, 84, 84), (1, 1, 1), 1), ((84, 85, 84), (0, 1, 1), 1)]


@pytest.mark.parametrize("precond", ["JACOBI", "NONE"])
@pytest.mark.parametrize("n,periodic,comps", CASES)
def test_one_launch_solve(n, periodic, comps, precond):
    ctx = D.Context(0)
    g = D.Grid(ctx, n, None, 2, periodic)
    s = D.MatrixSystem(g, components=comps)
    diag, rhs, x0 = _system(n, periodic, sum(n) + comps, comps)
    cells = int(np.prod(n))
    inter = lambda a: np.ascontiguousarray(np.moveaxis(a.reshape(a.shape[:-4] + (comps, cells)), -2, -1)
                                           .reshape(a.shape[:-4] + (comps * cells,)))
    s.set_coefficients(inter(diag), inter(rhs), inter(x0))
    solver = D.BiCGStab2({"Convergence Tolerance": 1e-11, "Maximum Iterations": 500, "tol_relative": 1}, precond=precond)
    launches = ctx.launch_count
    rep = solver.solve(s)
    launches = ctx.launch_count - launches
    assert rep["converged"], rep
    x = np.moveaxis(s.solution().reshape(cells, comps), -1, 0).reshape(rhs.shape)
    res = np.linalg.norm(rhs - _apply(diag, x, n, periodic)) / np.linalg.norm(rhs)
    assert res < 1.1e-11
    assert abs(rep["true_res_abs"] / rep["b_norm"] - res) < 1e-13
    assert (launches == 1) == (comps * cells < (590000 if precond == "JACOBI" else 515000)), launches
    if comps == 1 and cells < 5000:
        rp, cols, vals = diag_to_csr(len(n), n, diag[:, 0].reshape(7, -1), periodic)
        ox, info = O.bicgstab2(rp, cols, vals, rhs.reshape(-1), x0.reshape(-1), 1e-11 * np.linalg.norm(rhs), 500,
                               O.PREC_JACOBI if precond == "JACOBI" else O.PREC_NONE)
        assert rel_l2(x, ox) < 1e-9 and abs(rep["iters"] - info["iters"]) <= 2
