"""The column pass's long runs (large grids): velocities against the oracle on
sampled pixels, with flat frames and with frames whose values change by
decades row by row, and bands of a host call against one band.  Grids on both
sides of the rule's line (320,000 points of both frames)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


def frames(shape, steep):
    from pyflct_gb300 import synth
    rng = np.random.default_rng(shape[0])
    f1 = synth.kfield(shape, rng)
    f2 = synth.fourier_shift(f1, 0.3, -0.4)
    if steep:  # a decade every few rows, up and down: run units lie far apart
        k = 10.0 ** (8.0 * np.sin(np.arange(shape[0]) / 9.0))[:, None]
        f1, f2 = f1 * k, f2 * k
    return f1 + 3.0, f2 + 3.0


# 2 x 400 x 400 and 2 x 399 x 401 grid points: just at and just under
@pytest.mark.parametrize("shape", [(632, 633), (631, 631), (650, 701), (400, 400), (399, 401)])
@pytest.mark.parametrize("steep", [False, True])
def test_against_the_oracle_on_sampled_rows(shape, steep):
    import pyoracle as po
    from pyflct_gb300.flct import flct
    f1, f2 = frames(shape, steep)
    vx, vy, vm = flct(f1, f2, 1.0, 1.0, 3.0)
    # the oracle's windows of every 13th row and 11th column: the box around
    # a pixel, its own mean and Gaussian
    bad = 0
    for i in range(7, shape[0], 53):
        for j in range(5, shape[1], 37):
            g1, g2 = po.extract_window(f1, f2, i, j, sigma=3.0)
            sx, sy = po.cross_cor(g1, g2)[:2]
            d = max(abs(vx[i, j] - sy), abs(vy[i, j] - sx))
            bad += not d <= 1e-3
    # steep frames hold windows whose peak two FP32 spectra cannot tell apart
    assert bad <= (0 if not steep else 2), bad


@pytest.mark.parametrize("steep", [False, True])
def test_bands_equal_one_band(steep, monkeypatch):
    from pyflct_gb300 import _lib
    from pyflct_gb300.flct import make_params
    shape = (700, 640)
    f1, f2 = frames(shape, steep)
    p = make_params(1.0, 1.0, 3.0)
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    got = []
    for nb in ("0", "3"):
        monkeypatch.setenv("FLCT_HOST_BANDS", nb)
        ctx = _lib.Context(0)
        out = [np.empty(shape) for _ in range(3)]
        ctx.check(ctx.lib.flct_gpu_velocity(ctx.h, C.byref(p), ptr(f1), ptr(f2), *shape, *[ptr(o) for o in out]))
        got.append(out)
        ctx.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
