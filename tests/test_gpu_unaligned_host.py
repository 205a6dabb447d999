"""Host arrays that do not start on an 8-byte boundary (a view into a file's
bytes): the same fields as aligned ones, bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


def at(a, off):
    b = np.zeros(a.size * 8 + 16, np.uint8)
    v = b[(-b.ctypes.data) % 8 + off:][:a.size * 8].view(np.float64).reshape(a.shape)
    v[...] = a
    return v


def ptr(a):
    return C.cast(a.ctypes.data, C.POINTER(C.c_double))


@pytest.mark.parametrize("off", [1, 4])
def test_inputs_and_outputs(off):
    from pyflct_gb300 import _lib, synth
    from pyflct_gb300.flct import flct, make_params, shift_frac2d, warp_frac2d
    rng = np.random.default_rng(off)
    f1 = np.ascontiguousarray(synth.kfield((61, 53), rng))
    f2 = np.ascontiguousarray(synth.fourier_shift(f1, 0.4, -0.3))
    d = synth.smooth_shift(f1.shape, rng, rms=1.0)
    ctx = _lib.context(0)
    want = flct(f1, f2, 1.0, 1.0, 3.0)
    for got in (flct(at(f1, off), f2, 1.0, 1.0, 3.0), flct(f1, at(f2, off), 1.0, 1.0, 3.0)):
        assert all(np.array_equal(g, w) for g, w in zip(got, want))
    out = [at(np.zeros_like(f1), off) for _ in range(3)]
    p = make_params(1.0, 1.0, 3.0)
    ctx.check(ctx.lib.flct_gpu_velocity(ctx.h, C.byref(p), ptr(f1), ptr(f2), *f1.shape, *[ptr(o) for o in out]))
    assert all(np.array_equal(g, w) for g, w in zip(out, want))
    assert np.array_equal(shift_frac2d(at(f1, off), 0.7, -0.2), shift_frac2d(f1, 0.7, -0.2))
    assert np.array_equal(warp_frac2d(f1, at(d[0], off), d[1]), warp_frac2d(f1, *d))
