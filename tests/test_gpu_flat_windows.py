"""Windows and whole frames with one flat image: its transform is zero, so is the
correlation, and the shift is exactly 0 (as the oracle's), whatever the other
sub-image holds; its neighbours keep the results they have without it."""
import numpy as np
import pytest

import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


@pytest.mark.parametrize("n", [4, 8, 12, 16, 20, 24, 28, 32, 36, 40, 44, 48, 52, 56, 60, 64, 68, 84, 100, 128])
@pytest.mark.parametrize("kr", [None, 0.6])
def test_one_sub_image_zero(n, kr):
    from pyflct_gb300.flct import cross_cor
    rng = np.random.default_rng(n)
    g1 = rng.standard_normal((17, n, n))
    g2 = np.roll(g1, (1, 1), (1, 2)) + 0.1 * rng.standard_normal(g1.shape)
    wx, wy = cross_cor(g1, g2, kr=kr)
    z1, z2 = g1.copy(), g2.copy()
    z1[2] = z2[5] = z1[6] = z2[6] = z1[16] = 0.0
    z1[9], z2[9] = 0.0, g2[9] * 1e25
    z1[11], z2[11] = g1[11] * 1e-30, 0.0
    gx, gy = cross_cor(z1, z2, kr=kr)
    flat = [2, 5, 6, 9, 11, 16]
    ox, oy = po.cross_cor_batch(z1[flat], z2[flat], kr=kr)
    assert not ox.any() and not oy.any()
    assert not gx[flat].any() and not gy[flat].any()
    rest = [k for k in range(17) if k not in flat]
    assert np.array_equal(gx[rest], wx[rest]) and np.array_equal(gy[rest], wy[rest])


@pytest.mark.parametrize("sigma", [4.0, 5.0, 8.0, 12.0, 20.0])
@pytest.mark.parametrize("hires", [False, True])
def test_fields_over_a_hole_of_one_frame(sigma, hires):
    """A block of one frame is exactly zero, the other frame goes on: where the box lies inside it the velocity
    is the reference's for a zero correlation (0; with -h its search of an all-zero patch ends at -1)."""
    from pyflct_gb300 import synth
    from pyflct_gb300.flct import flct
    rng = np.random.default_rng(3)
    f1 = synth.kfield((150, 160), rng)
    f2 = synth.fourier_shift(f1, 0.3, -0.4)
    f1, f2 = f1.copy(), f2.copy()
    f1[10:130, 20:140] = 0.0
    vx, vy, vm = flct(f1, f2, 1.0, 1.0, sigma, hires=hires, skip="5")
    half = int(int(sigma) * np.sqrt(np.log(100.0))) // 2 * 2
    i, j = np.arange(0, 150, 5), np.arange(0, 160, 5)
    inside = np.ix_(i[(i - half >= 10) & (i + half + 1 <= 130)], j[(j - half >= 20) & (j + half + 1 <= 140)])
    ox, oy, om = po.velocity(f1, f2, sigma=sigma, hires=hires, skip=5)
    assert vx[inside].size and (ox[inside] == (-1 if hires else 0)).all()
    for a, b in ((vx, ox), (vy, oy), (vm, om)):
        assert np.array_equal(a[inside], b[inside])


@pytest.mark.parametrize("shape", [(16, 16), (97, 101), (300, 200), (3, 10007)])
@pytest.mark.parametrize("hires", [False, True])
@pytest.mark.parametrize("value", [0.0, 1.5])
def test_whole_frame_flat(shape, hires, value):
    """sigma = 0 with one frame flat (sums of 1.5 are exact)."""
    from pyflct_gb300.flct import flct
    f = np.random.default_rng(shape[1]).standard_normal(shape)
    for f1, f2 in ((np.full(shape, value), f), (f, np.full(shape, value)), (f * 0 + value, f * 0 - value)):
        got = [float(np.squeeze(a)) for a in flct(f1, f2, 1.0, 1.0, 0.0, hires=hires)]
        want = [-1.0, -1.0, 1.0] if hires else [0.0, 0.0, 1.0]
        assert got == want
        if max(shape) < 1000:  # (the oracle takes seconds a long line)
            assert want == [float(np.squeeze(a)) for a in po.velocity(f1, f2, sigma=0.0, hires=hires)]
