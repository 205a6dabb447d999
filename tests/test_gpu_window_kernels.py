"""The FP32 window kernels against the FP64 oracle at every box side a kernel
is compiled for, where their layouts change: each radix mix, each count of
lanes per window, scaled inputs, flat and non-finite windows.

Tolerance: the project's max |dv| <= 1e-3 px with its tie rule; FP32 transforms
of well-conditioned windows leave about 1e-5.
"""
import numpy as np
import pytest

import pyoracle as po
from _compare import TIE_REL, TOL

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


def windows(n, count, seed):
    """Pairs of windows displaced by up to a pixel or two, Gaussian-weighted as in the path."""
    from pyflct_gb300 import synth
    rng = np.random.default_rng(seed)
    g1, g2 = np.empty((count, n, n)), np.empty((count, n, n))
    w = np.exp(-(np.arange(n) - n / 2 + 1) ** 2 / (0.24 * n) ** 2)
    for k in range(count):
        f = synth.kfield((n + 8, n + 8), rng)
        s = synth.fourier_shift(f, *rng.uniform(-1, 1, 2))
        g1[k], g2[k] = (w[:, None] * w * x[4:4 + n, 4:4 + n] for x in (f, s))
    return g1, g2


def check(n, g1, g2, gx, gy, ox, oy, kr):
    d = np.maximum(np.abs(gx - ox), np.abs(gy - oy))
    for k in np.nonzero(~(d <= TOL))[0]:
        _, _, ab = po.cross_cor(g1[k], g2[k], kr=kr, want_abs=True)
        i, j = int(np.floor(gx[k] + n // 2 + 0.5)), int(np.floor(gy[k] + n // 2 + 0.5))
        near = any(0 <= i + a < n and 0 <= j + b < n and ab[i + a, j + b] >= (1 - TIE_REL) * ab.max()
                   for a in (-1, 0, 1) for b in (-1, 0, 1))
        assert near, (n, kr, int(k), float(d[k]))


@pytest.mark.parametrize("n", list(range(4, 129, 4)))
def test_every_box_side(n):
    from pyflct_gb300.flct import cross_cor
    # an odd count, more than the windows of one CTA at the small sides
    count = 67 if n <= 32 else 13
    g1, g2 = windows(n, count, 4000 + n)
    for kr in (None, 0.6):
        ox, oy = po.cross_cor_batch(g1, g2, kr=kr)
        gx, gy = cross_cor(g1, g2, kr=kr)
        check(n, g1, g2, gx, gy, ox, oy, kr)


@pytest.mark.parametrize("n", [4, 12, 16, 20, 24, 32, 36, 44, 48, 64, 68, 84, 100, 128])
def test_scaled_flat_and_nonfinite(n):
    from pyflct_gb300.flct import cross_cor
    g1, g2 = windows(n, 9, 5000 + n)
    s1, s2 = np.ones(9), np.ones(9)
    s1[1], s2[2], s1[3], s2[3], s1[4], s2[4] = 1e-30, 1e25, 1e-22, 1e28, 1e20, 1e20
    h1, h2 = g1 * s1[:, None, None], g2 * s2[:, None, None]
    h1[5] = h2[5] = 0.0       # flat: zero shift
    h1[6, n // 2, 1] = np.nan  # the reference's scan keeps a NaN first element: shift -n/2
    ox, oy = po.cross_cor_batch(h1, h2)
    gx, gy = cross_cor(h1, h2)
    keep = [k for k in range(9) if k != 6]
    check(n, h1[keep], h2[keep], gx[keep], gy[keep], ox[keep], oy[keep], None)
    assert gx[5] == 0.0 and gy[5] == 0.0
    assert np.array_equal(np.isnan([gx[6], gy[6]]), np.isnan([ox[6], oy[6]]))
    if not np.isnan(ox[6]):
        assert (gx[6], gy[6]) == (ox[6], oy[6])
