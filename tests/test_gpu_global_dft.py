"""The sigma = 0 mode over the sizes where its tiled direct DFTs change: one
tile, part tiles, each tile width, odd and prime sides; against the oracle
(the velocity tests' 1e-3 px).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


@pytest.mark.parametrize("shape", [(1, 1), (2, 3), (17, 64), (97, 101), (128, 300), (1009, 40), (330, 1000), (2048, 34)])
@pytest.mark.parametrize("kr", [None, 0.4])
def test_global_shift_sizes(shape, kr):
    import pyoracle as po
    from pyflct_gb300.flct import flct
    if kr and min(shape) < 2:
        pytest.skip("-k needs two points per axis")
    rng = np.random.default_rng(shape[0] * 7 + shape[1])
    f1 = rng.standard_normal(shape) if min(shape) < 16 else None
    if f1 is None:
        from pyflct_gb300 import synth
        f1 = synth.kfield(shape, rng)
        f2 = synth.fourier_shift(f1, *rng.uniform(-2, 2, 2))
    else:
        f2 = np.roll(f1, 1, 1)
    got = flct(f1, f2, 1.0, 1.0, 0.0, kr=kr)
    ref = po.velocity(f1, f2, sigma=0.0, **({"kr": kr} if kr else {}))
    for g, r in zip(got, ref):
        assert abs(float(np.squeeze(g)) - float(np.squeeze(r))) <= 1e-3, (shape, got, ref)


@pytest.mark.parametrize("shape", [(3, 10007), (9001, 4)])
def test_global_shift_long_lines(shape):
    """Long lines, few of them."""
    from pyflct_gb300.flct import flct
    rng = np.random.default_rng(shape[1])
    f1 = rng.standard_normal(shape)
    f2 = np.roll(f1, 3, int(shape[1] > shape[0]))
    vx, vy, vm = flct(f1, f2, 1.0, 1.0, 0.0)
    # white noise moved by whole pixels: a peak of one pixel, symmetric to the noise floor
    assert abs(float(np.squeeze(vx if shape[1] > shape[0] else vy)) - 3.0) < 0.2 and float(np.squeeze(vm)) == 1.0
