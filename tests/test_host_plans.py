"""The host's share of a shift or warp before the first launch: choosing a
line's transform is a lookup, whatever its length.  On the stand-in runtime,
without a GPU."""
import ctypes as C
import time

import numpy as np
import pytest

import _fake_cuda


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    h = _fake_cuda.Host(_fake_cuda.load(tmp_path_factory.mktemp("fake")))
    yield h
    h.close()


def quickest(host, name, nx, ny):
    a = [np.zeros((nx, ny)) for _ in range(4)]
    p = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in a]
    args = (p[0], C.c_double(0.5), C.c_double(0.25), p[1]) if name == "shift_frac2d" else p
    best = 1.0
    for _ in range(40):
        t = time.perf_counter()
        rc, _ = host.call(name, *args, nx, ny, 1)
        best = min(best, time.perf_counter() - t)
        assert rc == 0
    return best


# a search of the convolution's length took 0.2-1.1 ms at these, on each axis
@pytest.mark.parametrize("n", [1297, 2053, 4213, 5003])
@pytest.mark.parametrize("name", ["shift_frac2d", "warp_frac2d"])
def test_rough_lengths_cost_the_host_no_more(host, name, n):
    smooth = quickest(host, name, 3, 5120)  # a longer line without a convolution
    assert quickest(host, name, 3, n) <= smooth + 100e-6


@pytest.mark.parametrize("shape, lines", [((3, 37), False), ((17, 17), False), ((2, 17), False), ((37, 37), False),
                                          ((16, 36), True), ((3, 41), True), ((64, 17), True), ((17, 200), True)])
def test_small_warps_of_rough_sides_skip_the_convolutions(host, shape, lines):
    a = [np.zeros(shape) for _ in range(4)]
    rc, log = host.call("warp_frac2d", *[x.ctypes.data_as(C.POINTER(C.c_double)) for x in a], *shape, 1)
    assert rc == 0
    assert any("k_lines" in x for x in log) == lines and any("k_axis_fast" in x for x in log) != lines
