"""The line transforms behind the uniform shift and the warp's spectrum, over
the lengths where their passes change: each radix, mixed radices, lengths
with a large prime factor (chirp), the longest; against numpy's double
transforms.

Tolerances: those of the shift and velocity tests (4e-6 of max |image| at up
to 2048 points per axis; an FP32 transform's error grows with the square root
of its passes, far below that at 16384).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REL = 4e-6
PI = 3.1415926535898


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


def shifted(img, delx, dely):
    from pyflct_gb300.synth import make_freq
    n0, n1 = img.shape
    ph = np.exp(2j * PI * make_freq(n0)[:, None] * (-dely / n0)) * np.exp(2j * PI * make_freq(n1)[None, :] * (-delx / n1))
    return np.real(np.fft.ifft2(np.fft.fft2(img) * ph))


LENGTHS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 15, 16, 17, 31, 33, 97, 101, 169, 210, 221, 256, 257, 455, 1000,
           1009, 1200, 1536, 2039, 4096, 4099, 5000, 8191, 8192, 16384]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("axis", [0, 1])
def test_shift_line_length(n, axis):
    from pyflct_gb300.flct import shift_frac2d
    rng = np.random.default_rng(n)
    # 5 lines, or 300 (more than one round of short lines a CTA)
    m = 300 if n in (2, 16, 101) else 5
    img = rng.standard_normal((n, m) if axis == 0 else (m, n)) + 1.5
    dx, dy = rng.uniform(-7, 7, 2)
    got, ref = shift_frac2d(img, dx, dy, 1), shifted(img, dx, dy)
    err = np.abs(got - ref).max() / np.abs(img).max()
    assert err <= REL, (n, axis, err)
