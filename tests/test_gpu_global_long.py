"""The sigma = 0 mode on few, long lines, on both sides of its tiles' rules:
against numpy's double transforms, at the velocity tests' 1e-3 px."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def gpu():
    from pyflct_gb300 import _lib, build
    build.build()
    return _lib.context(0)


# 2432 / 2433: tiles of 8 lines; 9728 / 9729: one output a thread (3 lines: one round of blocks at 10007, 4: not)
@pytest.mark.parametrize("shape", [(3, 2432), (8, 2433), (9, 2433), (4, 9728), (3, 9729), (3, 10007), (4, 10007), (40, 3001)])
@pytest.mark.parametrize("turn", [False, True])
def test_shift_of_long_lines(shape, turn):
    from pyflct_gb300.flct import flct
    rng = np.random.default_rng(shape[1])
    # smooth along the line (three pixels), so that the peak is fitted on a rounded top; the lines differ
    x = np.fft.fft(rng.standard_normal(shape), axis=1)
    k = np.fft.fftfreq(shape[1])
    f1 = np.real(np.fft.ifft(x * np.exp(-2 * (np.pi * k * 3) ** 2), axis=1))
    f2 = np.real(np.fft.ifft(np.fft.fft(f1, axis=1) * np.exp(-2j * np.pi * k * 2.3), axis=1))
    c = np.real(np.fft.ifft2(np.conj(np.fft.fft2(f1 - f1.mean())) * np.fft.fft2(f2 - f2.mean())))
    c = np.abs(np.roll(c, (shape[0] // 2, shape[1] // 2), (0, 1)))
    i, j = np.unravel_index(c.argmax(), c.shape)
    assert 0 < i < shape[0] - 1 and 0 < j < shape[1] - 1
    v = c[i - 1:i + 2, j - 1:j + 2]
    fx, fy = 0.5 * (v[2, 1] - v[0, 1]), 0.5 * (v[1, 2] - v[1, 0])
    fxx, fyy = v[2, 1] + v[0, 1] - 2 * v[1, 1], v[1, 2] + v[1, 0] - 2 * v[1, 1]
    fxy = 0.25 * (v[2, 2] + v[0, 0] - v[2, 0] - v[0, 2])
    den = fxy * fxy - fxx * fyy
    slow, fast = i - shape[0] // 2 + (fyy * fx - fy * fxy) / den, j - shape[1] // 2 + (fxx * fy - fx * fxy) / den
    if turn:
        f1, f2, slow, fast = np.ascontiguousarray(f1.T), np.ascontiguousarray(f2.T), fast, slow
    vx, vy, vm = (float(np.squeeze(a)) for a in flct(f1, f2, 1.0, 1.0, 0.0))
    assert abs(vx - fast) <= 1e-3 and abs(vy - slow) <= 1e-3 and vm == 1.0
