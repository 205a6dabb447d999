"""The warp's tensor-core sum where its CTA plan changes: fewer pixel groups
than SMs, a last round cut into row chunks (and not), the last group partly
empty, several chunks with a short last one.  Same tolerance as the warp's
other tests (1e-6 of max |image|), against the double spectral sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PI = 3.1415926535898


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


def spectral(img, dfast, dslow):
    from pyflct_gb300.synth import make_freq
    n0, n1 = img.shape
    spec = np.fft.fft2(img) / img.size
    out = np.empty_like(img)
    for i in range(n0):
        xa = 2 * PI / n0 * (i - dslow[i])
        ya = 2 * PI / n1 * (np.arange(n1) - dfast[i])
        ey = np.exp(1j * ya[:, None] * make_freq(n1))
        ex = np.exp(1j * xa[:, None] * make_freq(n0))
        out[i] = ((ey @ spec.T) * ex).sum(1).real
    return out


# 256-pixel groups on 152 SMs: 38 of 76 (split would not help: one chunk), 2 chunks x 40 groups, 3 x 152 exactly,
# 3 x (152 + 3), 2 x 235 (83 left: two half rounds, no split), 5 chunks x 153
@pytest.mark.parametrize("shape", [(97, 200), (160, 64), (304, 128), (300, 133), (200, 300), (515, 76)])
def test_sum_over_tails(shape):
    from pyflct_gb300 import synth
    from pyflct_gb300.flct import warp_frac2d
    rng = np.random.default_rng(shape[0])
    img = synth.kfield(shape, rng)
    d = synth.smooth_shift(shape, rng, rms=1.5)
    for _ in range(2):  # the counts start from zero at every call
        err = np.abs(warp_frac2d(img, *d) - spectral(img, *d)).max() / np.abs(img).max()
        assert err <= 1e-6, (shape, err)
