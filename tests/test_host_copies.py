"""Which route a host array takes: a kernel that loads and stores its doubles
in place, or the runtime's copies.  On the stand-in runtime, without a GPU."""
import ctypes as C
import mmap

import numpy as np
import pytest

import _fake_cuda
from pyflct_gb300 import _lib
from pyflct_gb300.flct import make_params


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    h = _fake_cuda.Host(_fake_cuda.load(tmp_path_factory.mktemp("fake")))
    yield h
    h.close()


N = 72


def at(off):
    """N x N doubles, `off` bytes past a 16-byte boundary."""
    b = np.zeros(N * N * 8 + 32, np.uint8)
    a = (-b.ctypes.data) % 16 + off
    return b[a:a + N * N * 8].view(np.float64).reshape(N, N)


def ptr(a):
    return C.cast(a.ctypes.data, C.POINTER(C.c_double))


def routes(log):
    """(arrays copied by the kernel in, out), (by the runtime in, out)."""
    kern = [int(x.split()[3]) for x in log if "k_copy_arrays" in x]
    whole = [x.split() for x in log if x.startswith("copy ") and x.split()[2] == str(N * N * 8)]
    return kern, [sum(x[1] == k for x in whole) for k in "12"]


CALLS = {"velocity": (2, 3), "shift": (1, 1), "warp": (3, 1)}


def call(host, name, arrays):
    p = make_params(1.0, 1.0, 3.0)
    if name == "velocity":
        return host.call("velocity", C.byref(p), ptr(arrays[0]), ptr(arrays[1]), N, N, *[ptr(a) for a in arrays[2:]])
    if name == "shift":
        return host.call("shift_frac2d", ptr(arrays[0]), C.c_double(0.5), C.c_double(0.25), ptr(arrays[1]), N, N, 1)
    return host.call("warp_frac2d", *[ptr(a) for a in arrays], N, N, 1)


@pytest.mark.parametrize("name", CALLS)
def test_aligned_arrays_take_the_kernel(host, name):
    nin, nout = CALLS[name]
    for off in (0, 8):
        rc, log = call(host, name, [at(off) for _ in range(nin + nout)])
        assert rc == 0 and routes(log) == ([nin, nout], [0, 0])


@pytest.mark.parametrize("name", CALLS)
@pytest.mark.parametrize("off", [1, 2, 4, 12])
def test_unaligned_arrays_take_the_runtimes_copies(host, name, off):
    nin, nout = CALLS[name]
    for k in range(nin + nout):
        arrays = [at(off if q == k else 0) for q in range(nin + nout)]
        assert arrays[k].ctypes.data % 8
        rc, log = call(host, name, arrays)
        assert rc == 0
        # the side of the call that holds the array, all of it
        assert routes(log) == (([nout], [nin, 0]) if k < nin else ([nin], [0, nout])), k


def test_numpy_hands_unaligned_arrays_through():
    """Why the check is the library's: a view 4 bytes into a buffer is C-contiguous float64."""
    from pyflct_gb300.flct import _f64
    a = np.frombuffer(bytearray(8 * 100 + 4), np.float64, count=100, offset=4).reshape(10, 10)
    assert _f64(a).ctypes.data % 8 == a.ctypes.data % 8


def test_outputs_that_share_memory_are_written_in_order(host):
    """One scratch array for two results holds the later one, as copies one after another leave it."""
    f, g, a, b = (at(0) for _ in range(4))
    c = np.zeros(N * N + N)  # and two that overlap in part
    p = make_params(1.0, 1.0, 3.0)
    for out in ((a, a, b), (a, b, a), (b, a, a), (c[:N * N], a, c[N:])):
        rc, log = host.call("velocity", C.byref(p), ptr(f), ptr(g), N, N, *[ptr(o) for o in out])
        assert rc == 0 and routes(log) == ([2], [0, 3])
        assert [int(x.split()[3], 16) for x in log if x.startswith("copy 2 %d " % (N * N * 8))] == [o.ctypes.data for o in out]
    # neighbours do not
    rc, log = host.call("velocity", C.byref(p), ptr(f), ptr(f), N, N, ptr(c[:N * N]), ptr(a), ptr(b))
    assert rc == 0 and routes(log) == ([2, 3], [0, 0])
    whole = np.zeros((3, N, N))
    rc, log = host.call("velocity", C.byref(p), ptr(f), ptr(g), N, N, *[ptr(o) for o in whole])
    assert rc == 0 and routes(log) == ([2, 3], [0, 0])


@pytest.mark.parametrize("n, kernel", [(4, False), (32, False), (45, False), (46, True), (64, True)])
def test_small_copies_in_are_the_runtimes(host, n, kernel):
    """Up to 32 KB of inputs in all; results go by the kernel."""
    a = [np.zeros((n, n)) for _ in range(5)]
    rc, log = host.call("velocity", C.byref(make_params(1.0, 1.0, 0.0)), *[ptr(x) for x in a[:2]], n, n, *[ptr(x) for x in a[2:]])
    assert rc == 0
    copies = [x.split() for x in log if x.startswith("copy 1 ") and x.split()[2] == str(8 * n * n)]
    assert len(copies) == (0 if kernel else 2)
    assert [int(x.split()[3]) for x in log if "k_copy_arrays" in x] == ([2, 3] if kernel else [3])


READ_ONLY = """
import mmap, sys, ctypes as C, numpy as np
sys.path[:0] = %r
import _fake_cuda
from pyflct_gb300 import _lib
from pyflct_gb300.flct import make_params
lib = _lib.load(%r)
lib.fake_log.restype = C.c_char_p
lib.fake_reset.argtypes = [C.c_long]
host, (name, n, nin, nout, k) = _fake_cuda.Host(lib), %r
out = [np.zeros((n, n)) for _ in range(nout)]
out[k] = np.frombuffer(mmap.mmap(-1, 8 * n * n, prot=mmap.PROT_READ), np.float64).reshape(n, n)
p = [C.cast(a.ctypes.data, C.POINTER(C.c_double)) for a in [np.zeros((n, n)) for _ in range(nin)] + out]
if name == "velocity":
    rc, log = host.call("velocity", C.byref(make_params(1.0, 1.0, 3.0)), p[0], p[1], n, n, *p[2:])
elif name == "shift":
    rc, log = host.call("shift_frac2d", p[0], C.c_double(0.5), C.c_double(0.25), p[1], n, n, 1)
else:
    rc, log = host.call("warp_frac2d", *p, n, n, 1)
assert rc == _lib.ERR_CUDA, rc
assert sum("k_copy_arrays" in x for x in log) == (1 if 8 * n * n * nin > 32768 else 0)  # the inputs'
assert log[-1] == "sync stream"
"""


@pytest.mark.parametrize("name", CALLS)
@pytest.mark.parametrize("n", [N, 12])
def test_results_the_host_may_not_write_are_not_the_kernels(host, name, n):
    """A store of the kernel to a page without permission would be the device's fault.  The call
    ends with an error, or with the host's own fault where the results are less than a page."""
    import os
    import signal
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    nin, nout = CALLS[name]
    for k in range(nout):
        code = READ_ONLY % ([os.path.dirname(here), here], host.lib._name, (name, n, nin, nout, k))
        r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
        if 8 * n * n < mmap.PAGESIZE:
            assert r.returncode == -signal.SIGSEGV
        else:
            assert r.returncode == 0, r.stderr
