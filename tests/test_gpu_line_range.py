"""Uniform shifts of images near the ends of FP32's range and outside it: an image times a power of two gives the result times that power, bit for
bit (every step is exact in it while nothing leaves the range)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


# smooth lengths, powers of two, convolutions, short rough axes (no transforms), one line
@pytest.mark.parametrize("shape", [(200, 256), (100, 300), (257, 64), (1, 199), (16, 300), (256, 128), (53, 300), (1031, 40),
                                   (3, 8191), (2, 16384)])
@pytest.mark.parametrize("k", [-100, -58, 90, 118])
def test_shift_scales_exactly(shape, k):
    from pyflct_gb300.flct import shift_frac2d
    img = np.random.default_rng(shape[0] + shape[1]).standard_normal(shape)
    img[np.abs(img) < 1e-3] = 0.0  # a pixel's own bits stay normal floats at 2^-100
    want = shift_frac2d(img, 0.3, -0.7)
    got = shift_frac2d(img * 2.0 ** k, 0.3, -0.7)
    normal = np.abs(want) > 2.0 ** -20
    assert normal.mean() > 0.999
    assert np.array_equal(got[normal], want[normal] * 2.0 ** k)
    assert np.abs(got[~normal] - want[~normal] * 2.0 ** k).max(initial=0.0) <= 2.0 ** (k - 40)


def test_lines_of_unlike_size():
    """One huge line among small ones keeps them as well as the image's largest value allows."""
    from pyflct_gb300.flct import shift_frac2d
    img = np.random.default_rng(5).standard_normal((40, 300))
    img[7] *= 2.0 ** 120
    a, b = shift_frac2d(img, 1.0, 0.0), shift_frac2d(img, 0.4, 0.0)  # along the fast axis: lines stay apart
    assert np.isfinite(a).all() and np.isfinite(b).all()
    assert np.abs(a - np.roll(img, 1, 1)).max() <= 4e-6 * np.abs(img).max()


@pytest.mark.parametrize("k", [-1030, -200, 150, 1000])
def test_images_outside_fp32(k):
    """Doubles far outside FP32's range."""
    from pyflct_gb300.flct import shift_frac2d
    img = np.random.default_rng(2).integers(-1000, 1000, (60, 50)).astype(float)
    assert np.array_equal(shift_frac2d(np.ldexp(img, k), 2.4, 1.0), np.ldexp(shift_frac2d(img, 2.4, 1.0), k))


def test_in_place_and_beside_a_nan():
    """The image may be the result's own memory; one that is not finite keeps its NaN."""
    import ctypes as C
    from pyflct_gb300 import _lib
    from pyflct_gb300.flct import shift_frac2d
    img = np.random.default_rng(3).standard_normal((60, 50)) * 2.0 ** 120
    a, ctx = img.copy(), _lib.context(0)
    p = a.ctypes.data_as(C.POINTER(C.c_double))
    ctx.check(ctx.lib.flct_gpu_shift_frac2d(ctx.h, p, 0.3, -0.7, p, 60, 50, 1))
    assert np.array_equal(a, shift_frac2d(img, 0.3, -0.7)) and np.isfinite(a).all()
    img[4, 5] = np.nan
    assert np.isnan(shift_frac2d(img, 0.3, -0.7)).all()
    assert np.array_equal(shift_frac2d(np.zeros((60, 50)), 0.3, -0.7), np.zeros((60, 50)))
