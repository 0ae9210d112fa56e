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
