"""Local means of boxes above 64 x 64 on frames of one sign (an intensity image):
the exact sums of up to 124^2 values of nearly the largest magnitude."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


@pytest.mark.parametrize("sigma", [15.0, 16.5, 20.0, 28.0])
@pytest.mark.parametrize("offset", [1.95, -1.95, 1.2])
def test_offset_frames_against_the_oracle(sigma, offset):
    import pyoracle as po
    from pyflct_gb300 import synth
    from pyflct_gb300.flct import flct
    shape = (150, 170)
    rng = np.random.default_rng(3)
    f1 = synth.kfield(shape, rng)
    f2 = synth.fourier_shift(f1, 0.3, -0.4)
    f1, f2 = offset + 0.01 * f1, offset + 0.01 * f2
    vx, vy, vm = flct(f1, f2, 1.0, 1.0, sigma, skip="10")
    for i, j in ((0, 0), (40, 60), (70, 80), (80, 110), (140, 160)):
        g1, g2 = po.extract_window(f1, f2, i, j, sigma=sigma)
        sx, sy = po.cross_cor(g1, g2)[:2]
        assert abs(vx[i, j] - sy) <= 1e-3 and abs(vy[i, j] - sx) <= 1e-3, (i, j)
