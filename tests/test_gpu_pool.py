"""Device blocks kept between problems: a problem set up in the memory of
others, of other sizes, orders and precisions, or beside them in other threads,
gives the same fields bit for bit."""
import threading

import numpy as np
import pytest

import poremaps_gb300 as pm
from poremaps_gb300 import synth

pytestmark = pytest.mark.gpu

KINDS = [dict(precision="mixed"), dict(order="jacobi"), dict(order="redblack"),
         dict(order="reference"), dict(precision="mixed", kernel=1),
         dict(precision="mixed", kernel=13)]


def solve(shape, i, seed):
    g = synth.random_solid(shape, 0.3, seed)
    with pm.Problem(g, None, boundary_method=seed % 5, **KINDS[i]) as p:
        p.iterate(23)
        return p.fields()


def test_blocks_used_again():
    shapes = [(20, 21, 22), (23, 22, 21), (20, 21, 22), (9, 40, 33)]
    want = {}
    for turn in range(3):
        for k, shape in enumerate(shapes):
            for i in range(len(KINDS)):
                got = solve(shape, (i + turn) % len(KINDS), k)
                ref = want.setdefault((k, (i + turn) % len(KINDS)), got)
                assert all(np.array_equal(a, b) for a, b in zip(got, ref))


def test_blocks_of_several_threads():
    want = [solve((18, 20, 22), i, i) for i in range(len(KINDS))]
    bad = []

    def work(i):
        for _ in range(6):
            if not all(np.array_equal(a, b) for a, b in zip(solve((18, 20, 22), i, i), want[i])):
                bad.append(i)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(KINDS))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_release_memory():
    """Given back while a problem runs, and used again afterwards."""
    want = [solve((18, 20, 22), i, i) for i in range(len(KINDS))]
    g = synth.random_solid((18, 20, 22), 0.3, 0)
    with pm.Problem(g, None, boundary_method=0, **KINDS[0]) as p:
        p.iterate(11)
        pm.release_memory()
        got = [solve((18, 20, 22), i, i) for i in range(len(KINDS))]
        pm.release_memory()
        p.iterate(12)
        assert all(np.array_equal(a, b) for a, b in zip(p.fields(), want[0]))
    for a, b in zip(got, want):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
