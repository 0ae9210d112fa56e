"""Launch forms that the timings of one machine may never pick: every form gives
the same fields bit for bit, on lists shorter than a block, just longer than one
wave (3 CTAs of 256 on 152 SMs hold 116,736 voxels) and several waves long."""
import numpy as np
import pytest

import poremaps_gb300 as pm
from poremaps_gb300 import synth

pytestmark = pytest.mark.gpu

SHAPES = [((3, 4, 5), 0.2, 0), ((49, 49, 49), 0.0, 1), ((53, 90, 81), 0.3, 2),
          ((90, 80, 101), 0.25, 0)]


def fields(g, forms, **kw):
    pm.debug_launch_forms(*forms)
    try:
        with pm.Problem(g, None, **kw) as p:
            p.iterate(1)
            p.iterate(17)  # a captured block
            return p.fields()
    finally:
        pm.debug_launch_forms()


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("order,solver", [("jacobi", 2), ("jacobi", 3), ("redblack", 1),
                                          ("redblack", 2), ("redblack", 3)])
@pytest.mark.parametrize("shape,frac,bc", SHAPES)
def test_fp64_forms(order, solver, shape, frac, bc):
    g = synth.random_solid(shape, frac, 3)
    kw = dict(order=order, solving_algorithm=solver, boundary_method=bc)
    want = fields(g, (3, -1), **kw)
    for form in (0, 1, 2, -1):
        assert same(fields(g, (form, -1), **kw), want), form


@pytest.mark.parametrize("solver", [2, 3])
@pytest.mark.parametrize("shape,frac,bc", SHAPES)
def test_record_sweep_block_sizes(solver, shape, frac, bc):
    g = synth.random_solid(shape, frac, 3)
    kw = dict(precision="mixed", solving_algorithm=solver, boundary_method=bc)
    want = fields(g, (-1, -1), kernel=1, **kw)
    for variant in (0, 1, 2):
        for kernel in (13, -1):
            assert same(fields(g, (-1, variant), kernel=kernel, **kw), want), (variant, kernel)


def test_forms_that_do_not_exist():
    for bad in ((4, -1), (-2, -1), (-1, 3), (-1, -2)):
        with pytest.raises(pm.PMError):
            pm.debug_launch_forms(*bad)
