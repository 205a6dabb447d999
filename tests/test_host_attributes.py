"""A kernel's limit of dynamic shared memory belongs to the device, not to a
context: calls of several threads, each with a context of its own, share it.
So a call may only ever set a kernel's limit to one value, which covers every
launch.  On the stand-in runtime, without a GPU."""
import collections
import ctypes as C

import numpy as np
import pytest

import _fake_cuda


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    h = _fake_cuda.Host(_fake_cuda.load(tmp_path_factory.mktemp("fake")))
    yield h
    h.close()


# lines of each kernel and transform kind, chirps, and lengths without a plan (the axis kernels)
LENGTHS = [2, 16, 37, 53, 101, 2047, 2048, 2310, 3000, 4099, 6007, 8000, 8192, 8191, 8209, 9009, 10007, 16381, 16384]


def test_one_limit_per_kernel(host):
    limit, need = collections.defaultdict(set), collections.defaultdict(int)
    for nx, ny in [(n, 3) for n in LENGTHS] + [(4, n) for n in LENGTHS] + [(37, 53), (301, 8192)]:
        a = [np.zeros((nx, ny)) for _ in range(4)]
        p = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in a]
        for name, args in (("shift_frac2d", (p[0], C.c_double(0.5), C.c_double(0.25), p[1])), ("warp_frac2d", p)):
            rc, log = host.call(name, *args, nx, ny, 1)
            assert rc == 0
            for x in map(str.split, log):
                if x[0] == "attribute" and x[2] == "8":
                    limit[x[1]].add(int(x[3]))
                elif x[0] == "launch":
                    need[x[1]] = max(need[x[1]], int(x[-1]))
    assert sum("k_lines" in k for k in need) == 3 and sum("k_axis" in k for k in need) >= 4
    for k, v in limit.items():
        assert len(v) == 1, (k, sorted(v))
    for k, v in need.items():
        assert v <= max(limit.get(k, {0}) | {48 * 1024}), k
