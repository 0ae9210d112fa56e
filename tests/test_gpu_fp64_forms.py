"""The FP64 coefficient form over lists shorter and longer than a wave, with
every neighbourhood case and boundary method, against the oracle."""
import numpy as np
import pytest

import poremaps_gb300 as pm
from oracle.oracle import OracleProblem
from poremaps_gb300 import synth

pytestmark = pytest.mark.gpu


# 16 sweeps run as a captured block of overlapped launches.  Bound: 4e-13 of the
# field's largest value, some 25 roundings of 2^-53 a sweep over 17 sweeps (7e-14)
# times the sweeps' growth of a difference (below 5 over 17 sweeps).
@pytest.mark.parametrize("order", ["jacobi", "redblack"])
@pytest.mark.parametrize("shape,frac,bc", [((3, 4, 5), 0.2, 0), ((6, 5, 9), 0.5, 3),
                                           ((12, 11, 17), 0.35, 2), ((40, 70, 90), 0.3, 1),
                                           ((31, 33, 97), 0.6, 4)])
@pytest.mark.parametrize("solver", [2, 3])
def test_fp64_coefficient_form(order, shape, frac, bc, solver):
    g = synth.random_solid(shape, frac, 5 + bc)
    with pm.Problem(g, None, boundary_method=bc, solving_algorithm=solver, order=order) as pr:
        pr.iterate(1)
        pr.iterate(16)
        got = pr.fields()
    orc = OracleProblem(g, bc, solver)
    orc.iterate(17, order)
    f = orc.fields()
    for a, b in zip(got, (f.u, f.v, f.w, f.p)):
        assert np.abs(a - b).max() <= 4e-13 * max(np.abs(b).max(), 1e-300)
