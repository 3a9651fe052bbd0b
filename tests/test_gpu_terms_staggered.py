"""Composed functors on staggered grids: in one launch (up to eight terms) as in
a launch a term, to the bit."""
import numpy as np
import pytest

import dare_b200 as D
from tests.test_gpu_terms_fused import _build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,periodic,staggered,comps", [((20,), (0,), (1,), 3), ((20, 21), (0, 1), (1, 0), 1),
                                                        ((7, 34), (1, 0), (0, 1), 2), ((9, 8), (0, 0), (1, 1), 2)])
def test_one_launch_on_a_staggered_grid(n, periodic, staggered, comps):
    ctx = D.Context(0)
    dim = len(n)
    rng = np.random.default_rng(sum(n))
    g = D.Grid(ctx, n, None, 2, periodic, staggered=staggered)
    f = D.Field(g, 2, components=comps)
    f.upload(rng.normal(size=g.num_cells_ghosted * comps), 0)
    f.upload(rng.normal(size=g.num_cells_ghosted * comps), 1)
    faces = [D.DeviceArray(rng.uniform(-1.0, 1.0, size=g.face_shape(d))) for d in range(3)]
    terms = [D.Term("DDT", "SET", dt=1e-2), D.Term("CONVECTION", "ADD", face_vel=tuple(faces), limiter="VANLEER"),
             D.Term("DIFFUSION", "SUB", D=0.3), D.Term("CONVECTION", "SUB", vel=(0.3,) * dim, limiter="CDS")]
    bcs = [{2 * d + 1 + q: (1 + (q + c) % 2, 0.5 + c) for d in range(dim) if not periodic[d] for q in range(2)}
           for c in range(comps)]
    nothing = [D.Term("COEFFS", "ADD", coef=(None,) * 7)] * 6
    one = _build(g, f, terms, comps, bcs)
    many = _build(g, f, terms + nothing, comps, bcs)
    np.testing.assert_array_equal(one[0], many[0])
    np.testing.assert_array_equal(one[1], many[1])
    assert np.isfinite(one[0]).all() and np.abs(one[0][0]).min() > 0
