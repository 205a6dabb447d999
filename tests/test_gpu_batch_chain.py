"""Batches whose groups are single pairs (no prefix sums; one group: a chain of
dependent launches) against the same pairs called one by one: the same bits,
on first runs, on replays and after new inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


A = ((96, 131), dict(sigma=4.0))
B = ((64, 64), dict(sigma=8.0, thresh="0.1a", kr=0.5))
H = ((80, 77), dict(sigma=4.0, hires=True))
G = ((120, 140), dict(sigma=20.0, skip="4i"))
I = ((150, 90), dict(sigma=5.0, skip="3p1q2i", thresh=0.05))


@pytest.mark.parametrize("mix", [[A], [B], [H], [G], [I], [A, A], [A, B], [A, B, A], [G, H, I, A, A]],
                         ids=["a", "b", "hires", "big", "interp", "aa", "ab", "aba", "ghiaa"])
def test_equals_the_pairs_alone(mix):
    import torch
    from pyflct_gb300 import synth
    from pyflct_gb300.flct import FlctBatch, flct, make_params
    par = [{k: v for k, v in kw.items() if k != "sigma"} for _, kw in mix]
    params = [make_params(1.0, 1.0, kw["sigma"], **p) for (_, kw), p in zip(mix, par)]
    batch = FlctBatch([s for s, _ in mix], params)
    for rnd in range(2):
        rng = np.random.default_rng(rnd)
        frames = []
        for shape, _ in mix:
            f1 = synth.kfield(shape, rng)
            frames.append((f1, synth.fourier_shift(f1, 0.4, -0.3)))
        batch.load(frames)
        for _ in range(3):
            batch.run()
        torch.cuda.synchronize()
        for k, ((shape, kw), p) in enumerate(zip(mix, par)):
            ref = flct(*frames[k], 1.0, 1.0, kw["sigma"], **p)
            for got, want in zip((batch.vx[k], batch.vy[k], batch.vm[k]), ref):
                assert np.array_equal(got.cpu().numpy(), want)
