"""The reference order's kernels at the edges of their tiles and chunks, bit
for bit against the CPU oracle."""
import numpy as np
import pytest

import poremaps_gb300 as pm
from oracle.oracle import OracleProblem
from poremaps_gb300 import synth

pytestmark = pytest.mark.gpu


# the sweep's tiles hold 4 columns in y and 6 in z; x below, at and above its halo
@pytest.mark.parametrize("solver", [1, 2, 3])
@pytest.mark.parametrize("nx,ny,nz,bc", [(2, 3, 5, 3), (3, 4, 6, 4), (5, 5, 7, 0), (33, 8, 12, 1),
                                         (17, 9, 13, 2), (4, 23, 31, 0)])
def test_sweep_tiles(nx, ny, nz, bc, solver):
    g = synth.random_solid((nz, ny, nx), 0.3, 7 * nx + ny)
    orc = OracleProblem(g, bc, solver)
    with pm.Problem(g, None, boundary_method=bc, solving_algorithm=solver,
                    order="reference") as pr:
        for n in (1, 19):  # launched one by one, and as a captured block
            pr.iterate(n)
            orc.iterate(n, "reference")
            f = orc.fields()
            for a, b in zip(pr.fields(), (f.u, f.v, f.w, f.p)):
                assert np.array_equal(a, b)


# more tiles than are resident at once, with few voxels in x each
@pytest.mark.parametrize("nx,ny,nz,bc", [(1, 121, 130, 0), (2, 30, 601, 1), (3, 601, 30, 4)])
def test_sweep_many_thin_tiles(nx, ny, nz, bc):
    g = synth.random_solid((nz, ny, nx), 0.3, nx)
    orc = OracleProblem(g, bc, 2)
    orc.iterate(7, "reference")
    with pm.Problem(g, None, boundary_method=bc, order="reference") as pr:
        pr.iterate(7)
        got = pr.fields()
    f = orc.fields()
    for a, b in zip(got, (f.u, f.v, f.w, f.p)):
        assert np.array_equal(a, b)


def test_sweep_wait_runs_out():
    """With the test hook a tile gives up after its first look at a neighbour's
    values: the sweep ends, the call reports it, and the problem sweeps on."""
    g = synth.random_solid((14, 10, 12), 0.2, 3)
    with pm.Problem(g, None, order="reference") as pr:
        pm.debug_tma_fail(True)
        try:
            with pytest.raises(pm.PMError) as ei:
                pr.iterate(1)
                pr.fields()
        finally:
            pm.debug_tma_fail(False)
        assert ei.value.status == 3 and "timed out" in str(ei.value)
        pr.reset()
        pr.iterate(3)
        got = pr.fields()
    orc = OracleProblem(g, 0, 2)
    orc.iterate(3, "reference")
    f = orc.fields()
    for a, b in zip(got, (f.u, f.v, f.w, f.p)):
        assert np.array_equal(a, b)


def _values(kind, shape, rng):
    if kind == "zero":
        return np.zeros(shape)
    if kind == "one":  # exact, across binades
        return np.ones(shape)
    if kind == "ties":  # odd multiples of half a unit of sums above 2^20
        return rng.integers(-3, 9, shape) * 2.0 ** -33
    if kind == "positive":
        return rng.random(shape) ** 4
    if kind == "noise":  # sums near zero
        return rng.standard_normal(shape)
    # magnitudes far apart, subnormal numbers and both zeros among them
    a = rng.standard_normal(shape) * 2.0 ** rng.integers(-60, 10, shape)
    a[rng.random(shape) < 0.1] = -0.0
    a[rng.random(shape) < 0.05] = 5e-324
    return a


@pytest.mark.parametrize("kind", ["zero", "one", "ties", "positive", "noise", "mixed"])
@pytest.mark.parametrize("shape,box", [((7, 16, 18), None), ((8, 16, 16), (1, 14, 2, 12, 1, 6)),
                                       ((16, 20, 31), (0, 30, 0, 19, 3, 12))])
def test_serial_sums(kind, shape, box):
    """Permeability sums (2,016 to 9,920 voxels: below, at and above chunks of
    2,048) equal to the reference's voxel-by-voxel additions."""
    rng = np.random.default_rng(5)
    for solid in (0.0, 0.3):
        g = synth.random_solid(shape, solid, 9) if solid else np.zeros(shape, np.uint8)
        f = [_values(kind, shape, rng) for _ in range(4)]
        if kind == "ties":
            f[2][0, 0, 0] = 2.0 ** 20
        kw = {"dom_interest": (pm.C.c_int * 6)(*box)} if box else {}
        with pm.Problem(g, None, order="reference", voxel_size=1.0, porosity=0.5, **kw) as pr:
            pr.set_fields(*f)
            got = pr.permeability().as_dict()
        orc = OracleProblem(g, 0, 2, 1.0, porosity=0.5, **({"dom_interest": box} if box else {}))
        orc.set_fields(*f)
        want = orc.permeability()
        for k, v in got.items():
            if hasattr(want, k) and k not in ("iterations", "sweeps", "conv", "converged"):
                assert np.array_equal(v, getattr(want, k), equal_nan=True), k
