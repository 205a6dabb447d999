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
    assert quickest(host, name, 3, n) <= smooth + 60e-6
