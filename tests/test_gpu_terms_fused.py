"""A composed functor on 1-D and 2-D grids runs as one launch up to eight terms
and four components, and as one launch a term beyond: both give the same bits.
The longer list is the shorter one with COEFFS terms that add nothing."""
import numpy as np
import pytest

import dare_b200 as D

pytestmark = pytest.mark.gpu


def _build(g, f, terms, comps, bcs):
    s = D.MatrixSystem(g, components=comps)
    for c, bc in enumerate(bcs):
        for face, (kind, value) in bc.items():
            s.set_bc(face, kind, value, component=c)
    s.build(f, terms)
    return s.coefficients()


@pytest.mark.parametrize("n,periodic,comps", [((5,), (0,), 1), ((129,), (1,), 2), ((16, 8), (0, 1), 1),
                                              ((17, 23), (1, 0), 3), ((40, 33), (0, 0), 4)])
def test_one_launch_is_the_launches_one_by_one(n, periodic, comps):
    ctx = D.Context(0)
    dim = len(n)
    rng = np.random.default_rng(sum(n) + comps)
    g = D.Grid(ctx, n, None, 2, periodic)
    f = D.Field(g, 2, components=comps)
    f.upload(rng.normal(size=g.num_cells_ghosted * comps), 0)
    f.upload(rng.normal(size=g.num_cells_ghosted * comps), 1)
    faces = [D.DeviceArray(rng.uniform(-1.0, 1.0, size=g.face_shape(d))) for d in range(3)]
    diff = [D.DeviceArray(rng.uniform(0.5, 2.0, size=g.face_shape(d))) for d in range(3)]
    cells = [D.DeviceArray(rng.normal(size=g.num_cells)) for _ in range(8)]
    vel = tuple(float(v) for v in rng.uniform(-1.0, 1.0, size=dim))
    terms = [D.Term("DDT", "SET", dt=1e-2), D.Term("CONVECTION", "ADD", face_vel=tuple(faces), limiter="VANALBADA"),
             D.Term("DIFFUSION", "SUB", face_D=tuple(diff)), D.Term("CONVECTION", "SUB", vel=vel, limiter="MINMOD"),
             D.Term("COEFFS", "SUB", coef=tuple(cells[:7]), rhs=cells[7]),
             D.Term("DIFFUSION", "SUB", D=0.3, scheme="CRANK_NICHOLSON")]
    if comps > 1:   # a component of its own, and one that is started afresh alone
        terms += [D.Term("DDT", "ADD", component=comps - 1, dt=0.5), D.Term("DIFFUSION", "ADD", component=0, D=0.1)]
    bcs = [{2 * d + 1 + q: (1 + (q + c) % 2, 0.5 + c) for d in range(dim) if not periodic[d] for q in range(2)}
           for c in range(comps)]
    nothing = [D.Term("COEFFS", "ADD", coef=(None,) * 7)] * (9 - len(terms))
    one = _build(g, f, terms, comps, bcs)
    many = _build(g, f, terms + nothing, comps, bcs)
    np.testing.assert_array_equal(one[0], many[0])
    np.testing.assert_array_equal(one[1], many[1])
    assert np.isfinite(one[0]).all() and np.abs(one[0][0]).min() > 0
