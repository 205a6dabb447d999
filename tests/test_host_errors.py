"""A host-buffer call that returns an error has finished with the caller's
arrays: whichever runtime call fails, the stream is waited for before the
return when a copy kernel may still read or write them.  On the stand-in
runtime, without a GPU."""
import ctypes as C

import numpy as np
import pytest

import _fake_cuda
from pyflct_gb300 import _lib
from pyflct_gb300.flct import make_params


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return _fake_cuda.load(tmp_path_factory.mktemp("fake"))


N = 72
A = [np.zeros((N, N)) for _ in range(5)]
P = [a.ctypes.data_as(C.POINTER(C.c_double)) for a in A]
PAR = {"velocity": make_params(1.0, 1.0, 3.0), "interpolated": make_params(1.0, 1.0, 3.0, thresh="0.1", skip="3i"),
       "whole": make_params(1.0, 1.0, 0.0), "tuned": make_params(1.0, 1.0, 3.0, form="auto")}


def call(host, name, fail_at=0):
    if name == "shift":
        return host.call("shift_frac2d", P[0], C.c_double(0.5), C.c_double(0.25), P[1], N, N, 1, fail_at=fail_at)
    if name == "warp":
        return host.call("warp_frac2d", *P[:4], N, N, 1, fail_at=fail_at)
    return host.call("velocity", C.byref(PAR[name]), P[0], P[1], N, N, *P[2:], fail_at=fail_at)


@pytest.mark.parametrize("name", ["shift", "warp", *PAR])
def test_no_copy_outlives_an_error(lib, name):
    for n in range(1, 200):
        host = _fake_cuda.Host(lib)
        rc, log = call(host, name, n)
        failed = lib.fake_failed()
        host.close()
        if not failed:
            assert rc == _lib.OK and n > 15
            return
        copies = [k for k, x in enumerate(log) if "k_copy_arrays" in x and not x.endswith("FAILS")]
        waits = [k for k, x in enumerate(log) if x.startswith("sync stream") and not x.endswith("FAILS")]
        if copies and (rc != _lib.OK or not waits):
            assert waits and waits[-1] > copies[-1], (n, log)
    assert False, "the call never got through"
