"""Order in which the reference-order sweep's tiles are taken (pm_wave.h), on
the host: every tile once, none before the tiles it waits for, and tiles that are
resident together do not form a chain along a row, on which most of them would
only wait."""
import heapq
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ is missing")
    exe = str(tmp_path_factory.mktemp("wave") / "wave_tiles_check")
    subprocess.run([cxx, "-O1", "-std=c++17", os.path.join(HERE, "wave_tiles_check.cpp"), "-o",
                    exe], check=True)
    return exe


@pytest.mark.parametrize("ty,tz", [(1, 1), (1, 7), (9, 1), (2, 2), (3, 5), (5, 3), (12, 11),
                                   (250, 167), (128, 86), (400, 3)])
def test_tile_order(checker, ty, tz):
    out = subprocess.run([checker, str(ty), str(tz)], capture_output=True, text=True,
                         check=True).stdout.split()
    t = np.array(out, int).reshape(-1, 2)
    at = np.full((ty, tz), -1)
    at[t[:, 0], t[:, 1]] = np.arange(ty * tz)
    assert at.min() >= 0  # a permutation
    assert (at[1:, :] > at[:-1, :]).all() and (at[:, 1:] > at[:, :-1]).all()
    # `resident` tiles at a time, each a unit of time once what it waits for is
    # half done: the sweep takes no longer than the tiles' work shared evenly and
    # the longest chain of half steps one after the other.  (250 x 167 tiles: 215
    # units of 349 in this order, 6,408 in rows.)
    resident, done, free = 300, np.zeros((ty + 1, tz + 1)), []
    for n, (y, z) in enumerate(t):
        begin = heapq.heappop(free) if n >= resident else 0.0
        start = max(begin, done[y, z + 1] - 0.5, done[y + 1, z] - 0.5)
        done[y + 1, z + 1] = start + 1.0
        heapq.heappush(free, start + 1.0)
    bound = ty * tz / resident + 0.5 * (ty + tz) + 1.0
    assert done.max() <= bound, (done.max(), bound)
