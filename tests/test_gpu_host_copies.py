"""Host-buffer calls on pageable arrays: sizes on both sides of the copy
kernel's limit (16 MB an array), odd counts, starts 8 bytes off a 16-byte
boundary, outputs never touched before.  The fields are those of a
device-buffer call, bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


def at(n, off):
    """n float64 starting `off` doubles past a 16-byte boundary."""
    a = np.empty(n + 3)
    skip = (a.ctypes.data // 8) % 2
    return a[skip + off: skip + off + n]


def ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.mark.parametrize("shape", [(33, 41), (128, 128), (361, 363), (1447, 1449), (1450, 1450)])
@pytest.mark.parametrize("off", [0, 1])
def test_velocity_matches_device_call(shape, off):
    from pyflct_gb300 import _lib, synth
    from pyflct_gb300.flct import flct_batch, make_params
    rng = np.random.default_rng(shape[0] + off)
    f1 = synth.kfield(shape, rng)
    f2 = synth.fourier_shift(f1, 0.4, -0.3)
    p = make_params(1.0, 1.0, 3.0, kr=0.5, skip="5i" if min(shape) > 1000 else None)
    want, = flct_batch([(f1, f2)], [p])
    ctx = _lib.context(0)
    n = f1.size
    h = [at(n, off) for _ in range(2)]
    h[0][:], h[1][:] = f1.ravel(), f2.ravel()
    for _ in range(2):
        out = [at(n, off) for _ in range(3)]
        ctx.check(ctx.lib.flct_gpu_velocity(ctx.h, C.byref(p), ptr(h[0]), ptr(h[1]), *shape, *[ptr(o) for o in out]))
        for o, w in zip(out, want):
            assert np.array_equal(o.reshape(shape), w)


@pytest.mark.parametrize("shape", [(31, 37), (128, 96)])
def test_warp_from_odd_starts(shape):
    from pyflct_gb300 import _lib, synth
    from pyflct_gb300.flct import warp_frac2d
    rng = np.random.default_rng(shape[0])
    img = synth.kfield(shape, rng)
    d = synth.smooth_shift(shape, rng, rms=1.0)
    want = warp_frac2d(img, *d)
    ctx = _lib.context(0)
    h = [at(img.size, 1) for _ in range(3)]
    for a, b in zip(h, (img, *d)):
        a[:] = b.ravel()
    out = at(img.size, 1)
    ctx.check(ctx.lib.flct_gpu_warp_frac2d(ctx.h, *[ptr(a) for a in h], ptr(out), *shape, 1))
    assert np.array_equal(out.reshape(shape), want)
