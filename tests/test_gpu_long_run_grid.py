"""The column pass's long runs on coarse grids and for boxes above 64, and
beside short runs in one batch.

A frame whose grid takes long runs is compared with a band of its rows, cut at
a run's start, whose smaller grid takes short ones: windows that lie within the
band see the same pixels.  Where row sums lie far apart in size (steep frames)
a long run goes in pieces of a short one's length, with the same units: the
same bits.  Elsewhere a long run may drop low bits of values 2^54 times smaller than
its largest: the means agree to a float pair's last place, the fields far
within the project's 1e-3 px."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


def frames(shape, steep, seed):
    from pyflct_gb300 import synth
    rng = np.random.default_rng(seed)
    f1 = synth.kfield(shape, rng)
    f2 = synth.fourier_shift(f1, 0.3, -0.4)
    if steep:
        k = 10.0 ** (8.0 * np.sin(np.arange(shape[0]) / 9.0))[:, None]
        f1, f2 = f1 * k, f2 * k
    return f1 + 3.0, f2 + 3.0


# shape, sigma, -s, band of rows (starts at a multiple of 4 grid rows), box
CASES = [((1000, 1000), 6.0, 2, (304, 496), 24), ((1000, 1000), 16.0, 2, (304, 528), 68), ((420, 420), 20.0, 1, (96, 348), 84)]


@pytest.mark.parametrize("shape, sigma, skip, band, box", CASES)
@pytest.mark.parametrize("steep", [False, True])
def test_against_short_runs(shape, sigma, skip, band, box, steep):
    from pyflct_gb300.flct import flct
    points = lambda rows: 4 * (rows // skip) * (shape[1] // skip)
    line = 320000 * (skip + 1)
    assert points(shape[0]) >= line > points(band[1] - band[0]) and band[0] % (4 * skip) == 0
    f1, f2 = frames(shape, steep, shape[0] + int(sigma))
    s = str(skip) if skip > 1 else None
    full = flct(f1, f2, 1.0, 1.0, sigma, skip=s)
    part = flct(f1[band[0]:band[1]], f2[band[0]:band[1]], 1.0, 1.0, sigma, skip=s)
    lo, hi = band[0] + box, band[1] - box
    assert (hi - lo) // skip >= 40  # run boundaries at every place of a long run
    for a, b in zip(full, part):
        x, y = a[lo:hi], b[lo - band[0]:hi - band[0]]
        if steep:
            assert np.array_equal(x, y)
        else:
            assert np.abs(x - y).max() <= 1e-3


@pytest.mark.parametrize("order", [(0, 1, 2), (1, 0, 2), (2, 1, 0)])
def test_batch_of_long_and_short_runs(order):
    """Both column passes in one batch, in either order: the pairs' own results, bit for bit."""
    import torch
    from pyflct_gb300.flct import FlctBatch, flct, make_params
    mix = [((650, 520), 4.0, None), ((96, 131), 4.0, None), ((700, 700), 5.0, "3i")]
    mix = [mix[k] for k in order]
    batch = FlctBatch([m[0] for m in mix], [make_params(1.0, 1.0, m[1], skip=m[2]) for m in mix])
    pairs = [frames(m[0], k == 1, 7 + k) for k, m in enumerate(mix)]
    batch.load(pairs)
    for _ in range(3):
        batch.run()
    torch.cuda.synchronize()
    for k, m in enumerate(mix):
        want = flct(*pairs[k], 1.0, 1.0, m[1], skip=m[2])
        for got, w in zip((batch.vx[k], batch.vy[k], batch.vm[k]), want):
            assert np.array_equal(got.cpu().numpy(), w)
