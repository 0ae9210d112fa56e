"""The host runtime (problem set-up, kernel choice, device memory, the server's
rounds) on a stand-in for the device (fake_device.cpp): what reaches the device
in which order, with which buffers, and how much memory is held.  No GPU."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import poremaps_gb300 as pm

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "poremaps_gb300", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
GB = 1 << 30


@pytest.fixture(scope="session")
def built(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are missing")
    so = str(tmp_path_factory.mktemp("host") / "libhost.so")
    subprocess.run([cxx, "-O1", "-g", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic",
                    "-I", CUDA_INC,
                    os.path.join(HERE, "fake_device.cpp"), os.path.join(CSRC, "pm_api.cpp"),
                    os.path.join(CSRC, "pm_server.cpp"), "-lpthread", "-o", so], check=True)
    return so


class Host:
    """The library over the stand-in; a copy of its own for each test, since the
    kernel choices and kept blocks live as long as the library."""

    def __init__(self, so):
        L = self.L = C.CDLL(so)
        P, vp = C.POINTER, C.c_void_p
        L.pm_last_error.restype = C.c_char_p
        L.fake_trace.restype = C.c_char_p
        L.fake_used.restype = C.c_size_t
        L.fake_set_cost.argtypes = [C.c_char_p, C.c_double]
        L.fake_set_memory.argtypes = [C.c_int, C.c_size_t]
        L.pm_problem_create.argtypes = [P(pm.Params), vp, P(vp)]
        for f in ("pm_problem_destroy", "pm_server_destroy"):
            getattr(L, f).argtypes = [vp]
        L.pm_iterate.argtypes = [vp, C.c_int]
        L.pm_get_kernel.argtypes = [vp, P(C.c_int)]
        L.pm_problem_footprint.argtypes = [P(pm.Params), P(C.c_size_t)]
        L.pm_server_create.argtypes = [P(pm.ServerConfig), P(vp)]
        L.pm_server_submit.argtypes = [vp, P(pm.Params), vp, P(C.c_uint64)]
        L.pm_server_step.argtypes = [vp, P(C.c_int)]
        L.pm_server_poll.argtypes = [vp, P(pm.Completion), C.c_int, P(C.c_int)]
        L.pm_server_cancel.argtypes = [vp, C.c_uint64]

    def trace(self):
        t = self.L.fake_trace().decode().split("\n")
        self.L.fake_reset_trace()
        return t

    def params(self, shape, **kw):
        p = pm.Params()
        assert self.L.pm_params_default(C.byref(p)) == 0
        p.size[0], p.size[1], p.size[2] = shape
        for k, v in kw.items():
            setattr(p, k, v)
        return p

    def create(self, shape, fluid, **kw):
        """(status, handle); shape (nx, ny, nz), `fluid` fluid voxels."""
        p = self.params(shape, **kw)
        self.L.fake_set_fluid(fluid)
        geom = np.zeros(min(p.size[0] * p.size[1] * p.size[2], 1 << 20), np.uint8)
        h = C.c_void_p()
        return self.L.pm_problem_create(C.byref(p), geom.ctypes.data, C.byref(h)), h

    def kernel(self, h):
        k = C.c_int()
        assert self.L.pm_get_kernel(h, C.byref(k)) == 0
        return k.value


@pytest.fixture
def host(built, tmp_path):
    return Host(shutil.copy(built, tmp_path / "lib.so"))


def bad(trace):
    return [t for t in trace if t.startswith(("null", "unordered"))]


# ------------------------------------------------------------------ launch order
@pytest.mark.parametrize("kw", [dict(precision=1), dict(precision=1, kernel=13),
                                dict(order=pm.ORDER_JACOBI), dict(order=pm.ORDER_REDBLACK)])
def test_overlapped_sweeps_follow_their_set_up_data(host, kw):
    """Overlapped sweeps read records and list entries before they wait for the
    launch before them: what wrote these has to be ordered before that launch.
    Twice: the second problem finds the kernel choice made."""
    for _ in range(2):
        st, h = host.create((40, 40, 40), 20000, **kw)
        assert st == 0, host.L.pm_last_error()
        assert host.L.pm_iterate(h, 5) == 0
        t = host.trace()
        assert any(n in t for n in ("dc_inner_cr", "sweep64"))
        assert bad(t) == []
        host.L.pm_problem_destroy(h)


@pytest.mark.parametrize("it_eval", [1, 2, 10])
def test_server_sweeps_follow_their_set_up_data(host, it_eval):
    cfg = pm.ServerConfig(0, 0, 1, 0, 0, 0, 0)
    s = C.c_void_p()
    assert host.L.pm_server_create(C.byref(cfg), C.byref(s)) == 0
    host.L.fake_set_fluid(5000)
    geom = np.zeros(24 ** 3, np.uint8)
    p = host.params((24, 24, 24), it_eval=it_eval, max_iter=34)
    t = C.c_uint64()
    for _ in range(3):
        assert host.L.pm_server_submit(s, C.byref(p), geom.ctypes.data, C.byref(t)) == 0
    active = C.c_int(1)
    while active.value:
        assert host.L.pm_server_step(s, C.byref(active)) == 0, host.L.pm_last_error()
    assert bad(host.trace()) == []
    host.L.pm_server_destroy(s)


# ------------------------------------------------------------------ kernel choice
def test_choices_of_media_that_records_hold_and_do_not_hold(host):
    """Two media of one size and porosity on either side of the records' limit of
    2^27 - 1 fluid voxels: each gets the kernel chosen among its own candidates,
    over a store that exists, whichever comes first."""
    fits, not_fits, shape = (1 << 27) - 2, 1 << 27, (640, 640, 640)
    host.L.fake_set_cost(b"dc_inner_pf", 0.1)  # a kernel over the padded store wins
    seen = []
    for fluid in (not_fits, fits, not_fits, fits):
        st, h = host.create(shape, fluid, precision=1)
        assert st == 0, host.L.pm_last_error()
        assert host.L.pm_iterate(h, 3) == 0
        seen.append(host.kernel(h))
        assert bad(host.trace()) == []
        host.L.pm_problem_destroy(h)
    assert seen == [6, 13, 6, 13]


def forms(trace):
    return [int(t.split()[-1]) for t in trace if t.startswith("sweep64 form")]


@pytest.mark.parametrize("costs,want", [((1.0, 1.0, 1.0, 1.0), 3), ((1.0, 0.995, 0.992, 1.0), 3),
                                        ((1.0, 0.97, 0.98, 1.0), 1), ((1.0, 0.97, 0.96, 1.0), 2),
                                        ((0.9, 0.97, 0.96, 1.0), 0)])
@pytest.mark.parametrize("scale", [0.01, 1.0])
def test_fp64_form_is_timed(host, costs, want, scale):
    """The whole-stencil form unless another is at least 1 % faster; sweeps that
    take long are timed with fewer of them, and not one voxel per thread."""
    for i, c in enumerate(costs):
        host.L.fake_set_cost(b"sweep64 form %d" % i, c * scale)
    st, h = host.create((40, 40, 40), 20000, order=pm.ORDER_JACOBI)
    assert st == 0
    assert len(forms(host.trace())) <= (28 if scale < 0.1 else 9)
    assert host.L.pm_iterate(h, 2) == 0
    if scale == 1.0 and want == 0:
        want = 2
    assert forms(host.trace()) == [want, want]


# ------------------------------------------------------------------ device memory
def test_kept_blocks_of_another_device_are_not_free_here(host):
    """What destroyed problems left on another device does not count as free
    memory of this one."""
    L = host.L
    L.fake_set_memory(0, 200 << 20)
    L.pm_set_device(1)
    st, h = host.create((96, 96, 96), 400000, order=pm.ORDER_JACOBI)
    assert st == 0
    L.pm_problem_destroy(h)
    assert L.fake_used(1) > 60 << 20  # kept
    L.pm_set_device(0)
    host.trace()
    st, _ = host.create((150, 150, 150), 1000, order=pm.ORDER_JACOBI)  # 250 MB
    assert st == pm.PM_ERR_NOMEM
    assert b"needs" in L.pm_last_error() and "out of memory" not in host.trace()
    L.pm_set_device(1)  # there they do
    L.fake_set_memory(1, L.fake_used(1) + (2 << 20))
    st, h = host.create((96, 96, 96), 400000, order=pm.ORDER_JACOBI)
    assert st == 0, L.pm_last_error()
    L.pm_problem_destroy(h)


def test_server_budget_leaves_out_kept_blocks_of_another_device(host):
    L = host.L
    L.pm_set_device(1)
    st, h = host.create((160, 160, 160), 400000, order=pm.ORDER_JACOBI)
    assert st == 0
    L.pm_problem_destroy(h)
    L.pm_set_device(0)
    p = host.params((96, 96, 96), it_eval=10, max_iter=34, precision=0)
    need = C.c_size_t()
    assert L.pm_problem_footprint(C.byref(p), C.byref(need)) == 0
    L.fake_set_memory(0, int(1.7 * need.value))  # 0.8 of it holds one, not two
    L.fake_set_fluid(400000)
    cfg = pm.ServerConfig(0, 0, 0, 0, 0, 0, 0)
    s, t = C.c_void_p(), C.c_uint64()
    assert L.pm_server_create(C.byref(cfg), C.byref(s)) == 0
    geom = np.zeros(96 ** 3, np.uint8)
    for _ in range(2):
        assert L.pm_server_submit(s, C.byref(p), geom.ctypes.data, C.byref(t)) == 0
    active = C.c_int(1)
    while active.value:
        assert L.pm_server_step(s, C.byref(active)) == 0, L.pm_last_error()
    done, n = (pm.Completion * 2)(), C.c_int()
    assert L.pm_server_poll(s, done, 2, C.byref(n)) == 0
    assert n.value == 2 and [c.status for c in done] == [0, 0]
    L.pm_server_destroy(s)


def test_kept_blocks_are_bounded_and_given_back(host):
    """At most 1 GB is kept, the oldest blocks leave first, and
    pm_release_memory gives everything back."""
    L = host.L
    for n in (128, 150, 170, 190, 210, 256):
        hs = []
        for _ in range(3):
            st, h = host.create((n, n, n), 1000, order=pm.ORDER_JACOBI)
            assert st == 0, L.pm_last_error()
            hs.append(h)
        for h in hs:
            L.pm_problem_destroy(h)
        assert 0 < L.fake_used(0) <= GB
    assert L.pm_release_memory() == 0
    assert L.fake_used(0) == 0
    st, h = host.create((40, 40, 40), 1000, order=pm.ORDER_JACOBI)
    assert st == 0 and L.pm_release_memory() == 0 and L.fake_used(0) > 0  # in use: stays
    assert L.pm_iterate(h, 3) == 0
    L.pm_problem_destroy(h)


def test_problem_after_one_that_did_not_fit(host):
    """An allocation that failed is not reported by the launches of the next
    problem."""
    L = host.L
    p = host.params((128, 128, 128), order=pm.ORDER_JACOBI)
    need = C.c_size_t()
    assert L.pm_problem_footprint(C.byref(p), C.byref(need)) == 0
    # passes the check, which leaves out what alignment costs other problems
    L.fake_set_memory(0, need.value + (1 << 20))
    st, h = host.create((40, 40, 40), 1000, order=pm.ORDER_JACOBI)
    assert st == 0
    L.pm_problem_destroy(h)  # kept: counted as free, but not in one piece with the rest
    L.fake_split_memory(1)
    st, _ = host.create((128, 128, 128), 1000, order=pm.ORDER_JACOBI)
    assert st == pm.PM_ERR_NOMEM and b"out of memory" in L.pm_last_error()
    L.fake_split_memory(0)
    st, h = host.create((40, 40, 40), 1000, order=pm.ORDER_JACOBI)
    assert st == 0, L.pm_last_error()
    L.pm_problem_destroy(h)


@pytest.mark.parametrize("left", [0, 1 << 12])
def test_any_allocation_gets_what_is_kept(host, left):
    """Not only a problem's own buffers: where the server's tables do not fit
    beside the kept blocks, these are given back."""
    L = host.L
    cfg = pm.ServerConfig(GB, 0, 1, 0, 0, 0, 0)
    s, t = C.c_void_p(), C.c_uint64()
    assert L.pm_server_create(C.byref(cfg), C.byref(s)) == 0
    st, other = host.create((128, 128, 128), 1000, order=pm.ORDER_JACOBI)
    assert st == 0
    p = host.params((64, 64, 64), it_eval=10, max_iter=34, precision=1)
    L.fake_set_fluid(100000)
    geom = np.zeros(64 ** 3, np.uint8)
    st, h = host.create((64, 64, 64), 100000, precision=1, kernel=8, order=pm.ORDER_JACOBI)
    assert st == 0  # its blocks are what the request will use
    L.pm_problem_destroy(other)
    L.pm_problem_destroy(h)
    L.fake_set_memory(0, L.fake_used(0) + left)
    assert L.pm_server_submit(s, C.byref(p), geom.ctypes.data, C.byref(t)) == 0
    active = C.c_int(1)
    while active.value:
        assert L.pm_server_step(s, C.byref(active)) == 0, L.pm_last_error()
    done, n = (pm.Completion * 1)(), C.c_int()
    assert L.pm_server_poll(s, done, 1, C.byref(n)) == 0
    assert n.value == 1 and done[0].status == 0
    L.pm_server_destroy(s)


@pytest.mark.parametrize("nth", [1, 2, 5])
def test_failed_round_leaves_no_work_on_memory_that_is_kept(host, nth):
    """A launch that fails in the middle of a round: what was launched before it
    has ended when the call returns, so a cancelled sample's memory, which the
    next problem takes at once, is not in use."""
    L = host.L
    cfg = pm.ServerConfig(0, 0, 1, 0, 0, 0, 0)  # no graphs: launched one by one
    s, t = C.c_void_p(), C.c_uint64()
    assert L.pm_server_create(C.byref(cfg), C.byref(s)) == 0
    L.fake_set_fluid(5000)
    geom = np.zeros(24 ** 3, np.uint8)
    p = host.params((24, 24, 24), it_eval=10, max_iter=104)
    assert L.pm_server_submit(s, C.byref(p), geom.ctypes.data, C.byref(t)) == 0
    active = C.c_int()
    assert L.pm_server_step(s, C.byref(active)) == 0
    L.fake_fail_launch(nth)
    assert L.pm_server_step(s, C.byref(active)) == 3
    assert L.fake_pending() == 0
    assert L.pm_server_cancel(s, t) == 0
    L.pm_server_destroy(s)


# ------------------------------------------------------------------ problems beside each other
@pytest.mark.parametrize("n,fluid,order,want", [
    (128, 734000, pm.ORDER_REDBLACK, 3), (96, 500000, pm.ORDER_JACOBI, 3),  # beyond L2
    (56, 105000, pm.ORDER_JACOBI, 2), (56, 105000, pm.ORDER_REDBLACK, 2),  # more than a wave
    (24, 8300, pm.ORDER_JACOBI, 1), (48, 66000, pm.ORDER_REDBLACK, 1)])  # as alone
def test_fp64_forms_of_problems_that_share_the_device(host, n, fluid, order, want):
    """A group of three sweeps in the form that suits all three, whatever won
    alone; the same problems by themselves sweep as before."""
    L = host.L
    L.pm_block_group_timed.argtypes = [C.POINTER(C.c_void_p), C.c_int, C.c_int, C.c_int] + \
        [C.POINTER(C.c_double)] * 3
    L.fake_set_cost(b"sweep64 form 1", 0.9)
    hs = []
    for _ in range(3):
        st, h = host.create((n, n, n), fluid, order=order)
        assert st == 0
        hs.append(h)
    host.trace()
    for sweeps in (3, 20, 20):  # launched one by one, captured, replayed
        three = (C.c_void_p * 3)(*hs)
        assert L.pm_block_group_timed(three, 3, sweeps, 0, None, None, None) == 0
        assert set(forms(host.trace())) <= {want}
        assert L.pm_iterate(hs[0], sweeps) == 0
        assert set(forms(host.trace())) <= {1}
    for h in hs:
        L.pm_problem_destroy(h)
