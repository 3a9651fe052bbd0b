"""Host threads, each with a context of its own, solve systems of different size
at the same time.  The kernel is the same and its shared memory is not (57 and
30 KB a block), so what one thread sets up for its launch must not be what
another's launch is held to.  Every solve has to run, and to give the bits it
gives alone."""
import threading

import numpy as np
import pytest

import dare_b200 as D

pytestmark = pytest.mark.gpu

SIZES = [(25, 25, 25), (16, 16, 16)]


def _system(ctx, n):
    rng = np.random.default_rng(sum(n))
    g = D.Grid(ctx, n, None, 2, (1, 0, 1))
    s = D.MatrixSystem(g)
    diag = rng.uniform(-1.0, 0.2, size=(7, g.num_cells))
    diag[0] = 1.2 + np.abs(diag[1:]).sum(axis=0)
    s.set_coefficients(diag, rng.normal(size=g.num_cells))
    return s


def test_contexts_on_threads():
    threads = 4
    errors, start = [], threading.Barrier(threads)

    def work(q):
        try:
            s = _system(D.Context(0), SIZES[q % 2])
            zero = np.zeros(s.rows)
            full = D.BiCGStab2({"Convergence Tolerance": 1e-10, "Maximum Iterations": 200, "tol_relative": 1})
            short = D.BiCGStab2({"Convergence Tolerance": 1e-10, "Maximum Iterations": 1, "tol_relative": 1})
            s.set_initial_guess(zero)
            assert full.solve(s)["converged"]
            first = s.solution()
            start.wait()
            for _ in range(8):
                for _ in range(1000):
                    short.solve(s)
                s.set_initial_guess(zero)
                full.solve(s)
                assert np.array_equal(s.solution(), first)
        except Exception as e:
            errors.append(e)
            start.abort()

    pool = [threading.Thread(target=work, args=(q,)) for q in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not errors, [f"{type(e).__name__}: {e}"[:200] for e in errors]
