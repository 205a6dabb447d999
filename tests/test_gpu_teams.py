"""Windows per CTA: window counts below, at and above one CTA's teams and one
round of all CTAs give each window the result it has on its own (the same
bits), for every box side with shared CTA barriers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


@pytest.mark.parametrize("n", [12, 20, 24, 28, 36, 40, 44, 48, 52, 56, 60, 64])
def test_window_results_do_not_depend_on_their_number(n):
    from pyflct_gb300.flct import cross_cor
    rng = np.random.default_rng(n)
    g1 = rng.standard_normal((1100, n, n))
    g2 = np.roll(g1, (1, -2), (1, 2)) + 0.1 * rng.standard_normal(g1.shape)
    sx, sy = cross_cor(g1, g2)
    assert np.all(np.abs(sx - 1) < 0.6) and np.all(np.abs(sy + 2) < 0.6)
    for count in (1, 2, 3, 5, 6, 7, 8, 13, 1063, 1065):
        at = int(rng.integers(0, 1100 - count + 1))
        x, y = cross_cor(g1[at:at + count], g2[at:at + count])
        assert np.array_equal(x, sx[at:at + count]) and np.array_equal(y, sy[at:at + count])
