"""k_solution_to_field's rows, checked on the CPU (dare_b200/csrc/dare_core.cu).

A block takes a run of rows (i, j), a thread the same k of kSolRows of them at a
time; (i, j) is stepped by a block's rows with one wrap instead of a division a
row, and only cells near a periodic face write images.  This restates those
loops thread by thread and checks what tests/test_solution_to_field.py checks of
the pass: every access inside x and the ghosted field, no cell written twice,
and x and the field equal, cell for cell, to the three kernels' results and to
the oracle's CopyTo and ExchangeHaloCells.  Sizes: fewer rows than a block has,
rows of one cell, n1 = 1, n1 below and above a block's rows, and runs that end in
the middle of a thread's group."""
import itertools
import os
import re

import numpy as np
import pytest

from dare_b200.build import CSRC
from oracle import oracle as O
from tests.test_solution_to_field import CASES as SMALL
from tests.test_solution_to_field import block_shape, fused_ok, grid_dev, lin, three_kernels

with open(os.path.join(CSRC, "dare_core.cu")) as _f:
    ROWS = int(re.search(r"constexpr int kSolRows = (\d+);", _f.read()).group(1))


def by_rows(g, invd, x, num_sms):
    """The kernel, thread by thread; returns the writes it makes."""
    n0, n1, n2 = g["n"]
    ng, og, gn, per = g["ng"], g["og"], g["gn"], g["periodic"]
    hx, hy, hz = per[0], g["dim"] > 1 and per[1], g["dim"] > 2 and per[2]
    ncell, nghost = n0 * n1 * n2, gn[0] * gn[1] * gn[2]
    bx, by = block_shape(g)
    rows = n0 * n1
    grid = max(1, min(-(-rows // by), num_sms * 8))
    run = -(-rows // grid)
    stride = (gn[1] * gn[2], gn[2], 1)
    di, dj = by // n1, by % n1
    xw, fw = {}, {}

    def write(at, v):
        assert 0 <= at < nghost and at not in fw
        fw[at] = v

    for b, ty, tx in itertools.product(range(grid), range(by), range(bx)):
        ra, rb = b * run, min(b * run + run, rows)
        if ra >= rb:
            continue
        r = ra + ty
        i, j = r // n1, r % n1
        while r < rb:
            for k in range(tx, n2, bx):
                iu, ju = i, j
                hk = hz and (k < ng or k >= n2 - ng)
                for u in range(ROWS):
                    row = r + u * by
                    if row < rb:
                        assert (iu, ju) == (row // n1, row % n1)
                        c = row * n2 + k
                        assert 0 <= c < ncell and c not in xw
                        v = invd[c] * x[c] if invd is not None else x[c]
                        xw[c] = v
                        at = ((iu + og[0]) * gn[1] + ju + og[1]) * gn[2] + k + og[2]
                        write(at, v)
                        if hk or (hx and (iu < ng or iu >= n0 - ng)) or (hy and (ju < ng or ju >= n1 - ng)):
                            for d, q in enumerate((iu, ju, k)):
                                if d >= g["dim"] or not per[d]:
                                    continue
                                if q < ng:
                                    write(at + g["n"][d] * stride[d], v)
                                if q >= g["n"][d] - ng:
                                    write(at - g["n"][d] * stride[d], v)
                    iu, ju = iu + di, ju + dj
                    if ju >= n1:
                        iu, ju = iu + 1, ju - n1
            for _ in range(ROWS):
                i, j = i + di, j + dj
                if j >= n1:
                    i, j = i + 1, j - n1
            r += ROWS * by
    assert len(xw) == ncell
    return xw, fw


CASES = SMALL + [(1, (700,), 2, (1,)), (2, (300, 3), 2, (1, 1)), (2, (3, 300), 2, (0, 1)), (3, (40, 3, 2), 2, (1, 1, 0)),
                 (3, (5, 70, 3), 2, (1, 1, 1)), (3, (9, 11, 130), 2, (1, 0, 1))]


@pytest.mark.parametrize("num_sms", [1, 3, 148])
@pytest.mark.parametrize("dim,n,ng,periodic", CASES)
@pytest.mark.parametrize("jacobi", [True, False])
def test_rows_write_what_the_three_kernels_wrote(dim, n, ng, periodic, jacobi, num_sms):
    g = grid_dev(dim, n, ng, periodic)
    assert fused_ok(g)
    rng = np.random.default_rng(dim * 100 + sum(n) + ng)
    x = rng.normal(size=int(np.prod(g["n"])))
    invd = rng.uniform(0.5, 2.0, size=x.size) if jacobi else None
    phi0 = rng.normal(size=int(np.prod(g["gn"])))   # the field before: stale values everywhere
    xw, fw = by_rows(g, invd, x, num_sms)
    x_new, phi = x.copy(), phi0.copy()
    x_new[list(xw)] = list(xw.values())
    phi[list(fw)] = list(fw.values())
    x_ref, phi_ref = three_kernels(g, invd, x, phi0)
    np.testing.assert_array_equal(x_new, x_ref)
    np.testing.assert_array_equal(phi, phi_ref)
    og = O.make_grid(dim, n, None, ng, periodic)
    phi_o = phi0.copy()
    O.copy_to_field(og, x_ref, phi_o)
    O.exchange_halo(og, phi_o)
    np.testing.assert_array_equal(phi, phi_o)
