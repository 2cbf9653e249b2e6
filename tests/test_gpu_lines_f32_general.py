"""The general FP32 line kernel against numpy's FFT in double, at every radix of
its plans, one to six passes, lengths with and without padding words, and line
counts that leave a partial tile.  An FFT in FP32 is off by eps log2(n) of a
line's norm times the largest multiplier; the tolerance is ten times that."""
import numpy as np
import pytest

from fug30v0kxc_gb300.params import convection_params
from fug30v0kxc_gb300.solver import P3D
from tests.test_gpu_lines_f64 import _ref

pytestmark = pytest.mark.gpu
D1, D2, DEALIAS, FWD, INV = 1, 2, 3, 4, 5
EPS = 2.0 ** -23


@pytest.mark.parametrize("n", [4, 6, 8, 10, 16, 18, 30, 32, 48, 54, 60, 80, 90, 100, 150, 240, 250, 360, 480, 640, 1000, 1500,
                               2000, 2048])
def test_lengths(n, monkeypatch):
    monkeypatch.setenv("VEC_GENERIC_LINES", "1")
    rng = np.random.default_rng(n)
    for nx, ny, axis in ((n, 18, 2), (18, n, 1)):
        g = P3D(convection_params(nx, ny, 6))
        d = 0 if axis == 2 else 1
        f = rng.standard_normal((6, ny, nx)).astype(np.float32)
        f[1] = 0.0
        f[2] *= 1e3
        x = f.astype(np.float64)

        def close(got, want, order):
            kmax = (np.pi * n / 4.0) ** order
            tol = 10 * EPS * (1 + np.log2(n)) * kmax * np.abs(x).max(axis=(1, 2), keepdims=True) * np.sqrt(2.0)
            assert (np.abs(got - want) <= tol).all(), (n, axis, order)

        a, b = g.line_f32(d, D1, f, D2)
        close(a, _ref(x, axis, 1), 1)
        close(b, _ref(x, axis, 2), 2)
        assert np.array_equal(a, g.line_f32(d, D1, f))
        F = np.fft.rfft(x, axis=axis)
        k = np.arange(n // 2 + 1)
        keep = (k < n // 2 - (n // 2) // 3).reshape([-1 if q == axis else 1 for q in range(3)])
        close(g.line_f32(d, DEALIAS, f), np.fft.irfft(F * keep, n=n, axis=axis), 0)
        h = g.line_f32(d, FWD, f)
        re, im = F.real, np.flip(np.take(F.imag, np.arange(1, n // 2), axis=axis), axis=axis)
        assert np.abs(h - np.concatenate([re, im], axis=axis)).max() <= 10 * EPS * (1 + np.log2(n)) * n ** 0.5 * 5e3
        r, dr = g.line_f32(d, INV, h, D1)
        close(r, x, 0)
        close(dr, _ref(x, axis, 1), 1)
        g.close()
