"""The server's persistent round over its tile queue (k_batch_inner_round) and its
autotuner.  A server takes them where a launch shape is set and where the packed
records do not hold a sample (rows of 8,192 voxels and more), else the flat
sweeps: each test checks by the launches of a block that its path is the one that
ran.  Results are equal bit for bit."""
import numpy as np
import pytest

import poremaps_gb300 as pm
from poremaps_gb300 import synth

pytestmark = pytest.mark.gpu

BLOCK = 20
KW = dict(boundary_method=0, solving_algorithm=2, eps=1e-30, it_eval=BLOCK, it_write=BLOCK,
          max_iter=1061)
ROUND = 4  # residual, persistent round, correction, sums
SWEEPS = 3 + BLOCK - 1  # residual, one launch per sweep, correction, sums
FIELDS = ("wk13", "wk23", "wk33", "wmax_velz", "iterations", "sweeps")


def run(geoms, shape=None, **server):
    """Results by request, the launches of the first step and of the second (one
    block), and the launch shape at the end."""
    s = pm.Server(precision="mixed", **server)
    if shape:
        s.set_launch_shape(*shape)
    tickets = [s.submit(g, **KW) for g in geoms]
    launches, done = [], {}
    for _ in range(2):
        n = pm.kernel_launches()
        s.step()
        launches.append(pm.kernel_launches() - n)
    while s.step():
        pass
    done = {c.ticket: c for c in s.poll()}
    picked = s.launch_shape()
    s.close()
    assert all(done[t].status in (0, 5) for t in tickets)
    return [done[t].result for t in tickets], launches, picked


def same(a, b):
    return all(np.array_equal(getattr(x, f), getattr(y, f), equal_nan=True)
               for x, y in zip(a, b) for f in FIELDS)


@pytest.fixture(scope="module")
def small():
    return [synth.random_solid(s, 0.3, i) for i, s in
            enumerate([(12, 16, 20), (24, 20, 16), (9, 9, 9), (1, 1, 257), (40, 36, 44)])]


@pytest.mark.parametrize("shape", [(8192, 4, 256, 256), (512, 8, 128, 128)])
@pytest.mark.parametrize("use_graphs", [1, 0])
def test_persistent_round(small, use_graphs, shape):
    a, la, _ = run(small, shape=shape, use_graphs=use_graphs)
    b, lb, _ = run(small, use_graphs=use_graphs, relaunch_sweeps=1)
    c, lc, _ = run(small, use_graphs=use_graphs)
    assert (la[1], lb[1], lc[1]) == (ROUND, SWEEPS, SWEEPS)
    assert same(a, b) and same(c, b)


def test_autotuned_round():
    """Samples that the records do not hold: the round's shape is timed once and
    found again by the next server."""
    geoms = [synth.random_solid(s, 0.25, i) for i, s in
             enumerate([(3, 5, 8192), (2, 3, 9001), (4, 6, 8300)])]
    a, la, shape = run(geoms)
    assert la[1] == ROUND and tuple(shape.values()) == (8192, 4, 256, 256)
    b, lb, picked = run(geoms, autotune=1)
    assert lb[1] == ROUND and lb[0] > la[0]  # the first step timed candidates
    assert picked["item_voxels"] in (2048, 8192, 32768)
    assert (picked["round_threads"], picked["round_ctas_per_sm"]) in (
        (256, 2), (256, 3), (256, 4), (128, 4), (128, 6), (128, 8))
    c, lc, again = run(geoms, autotune=1)
    assert again == picked and lc[0] == la[0]
    assert same(a, b) and same(a, c)
