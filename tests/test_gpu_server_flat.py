"""The server's correction sweeps over flat items of 256 fluid voxels: samples
below, at and above one item, more items than a block stages at once, more than
one group of samples, and both solvers in one launch give the lone solve's
results bit for bit."""
import numpy as np
import pytest

import poremaps_gb300 as pm
from poremaps_gb300 import synth

pytestmark = pytest.mark.gpu

KW = dict(eps=1e-6, it_eval=10, max_iter=34, boundary_method=0)


def lone(g, solver):
    # iteration 0, then blocks of it_eval: the server's schedule of corrections
    with pm.Problem(g, None, precision="mixed", mixed_inner=10, order="jacobi",
                    solving_algorithm=solver, **KW) as p:
        return p.solve()


@pytest.mark.parametrize("shapes", [[(5, 3, 17), (4, 8, 8), (1, 1, 257), (6, 7, 9)],
                                    [(180, 176, 178), (8, 8, 9)],
                                    [(112, 110, 111), (108, 112, 113), (9, 30, 31)]])
def test_flat_items(shapes):
    # the last shape of each set is a random medium, the others are all fluid
    geoms = [np.zeros(s, np.uint8) for s in shapes[:-1]]
    geoms.append(synth.random_solid(shapes[-1], 0.3, 4))
    solvers = [2 + i % 2 for i in range(len(geoms))]
    s = pm.Server(precision="mixed")
    at = {s.submit(g, solving_algorithm=sv, **KW): i
          for i, (g, sv) in enumerate(zip(geoms, solvers))}
    out, active = {}, 1
    while active:
        active = s.step()
        for c in s.poll():
            out[at[c.ticket]] = c
    s.close()
    for i, (g, sv) in enumerate(zip(geoms, solvers)):
        want = lone(g, sv)
        got = out[i].result
        for f in ("wk13", "wk23", "wk33", "wmax_velz", "wmean_velz", "sweeps"):
            assert np.array_equal(getattr(got, f), getattr(want, f), equal_nan=True), (i, f)
