"""Row bands of a call on page-locked buffers: a frame with few rows keeps as
many as its column pass's runs allow.  On the stand-in runtime, without a GPU."""
import ctypes as C

import numpy as np
import pytest

import _fake_cuda
from pyflct_gb300.flct import make_params


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    h = _fake_cuda.Host(_fake_cuda.load(tmp_path_factory.mktemp("fake")))
    yield h
    h.close()


# short runs of 4 grid rows below 160,000 grid points (every pixel), else runs of 16
@pytest.mark.parametrize("shape, sigma, run, bands", [((100, 1000), 4.0, 4, 5), ((100, 2500), 4.0, 16, 5),
                                                      ((60, 4000), 5.0, 16, 3), ((90, 1800), 3.0, 16, 5),
                                                      ((400, 400), 4.0, 16, 5), ((24, 9000), 3.0, 16, 1)])
def test_bands_of_few_rows(host, shape, sigma, run, bands):
    nx, ny = shape
    a = [np.zeros(shape) for _ in range(5)]
    p = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in a]
    host.lib.fake_pinned(1)
    try:
        rc, log = host.call("velocity", C.byref(make_params(1.0, 1.0, sigma)), p[0], p[1], nx, ny, *p[2:])
    finally:
        host.lib.fake_pinned(0)
    assert rc == 0
    # the rows each band completes, by its copies out of vx
    base = a[2].ctypes.data
    out = [(int(x.split()[3], 16) - base, int(x.split()[2])) for x in log if x.startswith("copy 2 ")]
    out = sorted((o // (8 * ny), n // (8 * ny)) for o, n in out if 0 <= o < nx * ny * 8)
    if bands == 1:
        assert any("k_copy_arrays" in x for x in log) and not out
        return
    assert len(out) == bands
    assert [o for o, _ in out] == list(np.cumsum([0] + [n for _, n in out]))[:-1] and sum(n for _, n in out) == nx
    assert all(o % run == 0 for o, _ in out)


@pytest.mark.parametrize("sigma, n", [(4.0, 16), (8.0, 32)])
def test_bands_launch_the_light_shape(host, sigma, n):
    """One set of windows per CTA: few of them, and none of the tables that pay over many sets."""
    shape = (200, 250)
    a = [np.zeros(shape) for _ in range(5)]
    p = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in a]
    host.lib.fake_pinned(1)
    try:
        rc, log = host.call("velocity", C.byref(make_params(1.0, 1.0, sigma)), p[0], p[1], *shape, *p[2:])
    finally:
        host.lib.fake_pinned(0)
    assert rc == 0
    wins = [x.split() for x in log if x.startswith("launch") and "k_window_fp32ILi%d" % n in x]
    assert len(wins) == 5
    for x in wins:
        teams = int(x[5]) // n
        assert teams == 4 and int(x[-1]) < teams * n * (n + 2) * 8  # rows n + 1 apart, no copies of the weights
