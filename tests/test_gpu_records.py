"""The correction sweep over packed records (kernel 13, and what problems and
the server run by themselves) at the edges of the record format: rows of 8,191
voxels (the longest it holds) and 8,192 (the sweep then reads full slots),
periodic y faces of planes of more than 32,767 fluid voxels (absolute y
positions), periodic z faces, axes of length 1, wall faces, lists shorter than
a block.  The values are those of the fluid-list gather over the padded store
(kernel 1) bit for bit; no tolerance is involved."""
import numpy as np
import pytest

import poremaps_gb300 as pm
from poremaps_gb300 import synth

pytestmark = pytest.mark.gpu

SHAPES = [((3, 260, 260), 0), ((2, 3, 8191), 0), ((2, 3, 8192), 0), ((1, 1, 5), 0),
          ((5, 1, 300), 2), ((33, 40, 31), 1), ((9, 31, 64), 4)]


def fields(g, bc, solver, kernel):
    with pm.Problem(g, None, boundary_method=bc, solving_algorithm=solver, precision="mixed",
                    kernel=kernel, mixed_inner=30) as p:
        p.iterate(71)
        return p.fields()


@pytest.mark.parametrize("shape,bc", SHAPES)
@pytest.mark.parametrize("solver", [2, 3])
def test_records_equal_the_padded_store(shape, bc, solver):
    g = synth.random_solid(shape, 0.25, sum(shape) + bc)
    want = fields(g, bc, solver, 1)
    for kernel in (13, -1):
        for a, b in zip(fields(g, bc, solver, kernel), want):
            assert np.array_equal(a, b), (kernel, float(np.abs(a - b).max()))


@pytest.mark.parametrize("shape,bc", [((3, 260, 260), 0), ((2, 3, 8192), 0), ((20, 17, 33), 2)])
def test_server_records_equal_a_lone_solve(shape, bc):
    """The server packs the slots in place (or keeps them where they do not
    fit); its results are those of a lone solve, also over iterations that end
    inside a block."""
    g = synth.random_solid(shape, 0.25, sum(shape) + bc)
    kw = dict(boundary_method=bc, solving_algorithm=2, max_iter=1130, eps=1e-30)
    with pm.Problem(g, None, precision="mixed", kernel=1, **kw) as p:
        r = p.solve()
    with pm.Server("mixed") as s:
        s.submit(g, **kw)
        while s.step():
            pass
        (c,) = s.poll()
    assert c.status in (0, 5)
    for f in ("wk13", "wk23", "wk33", "wmax_velz", "iterations", "sweeps"):
        a, b = getattr(c.result, f), getattr(r, f)
        assert a == b or (a != a and b != b), f
