"""The FP64 line operators (64-bit fixed point inside, one exponent per pair of
lines) against numpy's FFT in double.

Lengths: every radix the plan takes (8, 6, 5, 4, 3, 2), one to six passes, the
smallest and largest length, lengths that are no multiple of 8, and line
counts that leave a partial tile.  Scales: fields near the ends of the double
range, subnormals, a large constant plus little, one spike, lines of very
different size next to each other.  numpy's own error is eps log2(n) of a
line's norm times the largest multiplier, and the tolerance ten times that.
"""
import numpy as np
import pytest

from fug30v0kxc_gb300.params import convection_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


def _ref(f, axis, order, length=4.0):
    n = f.shape[axis]
    sh = [-1 if a == axis else 1 for a in range(3)]
    k = (2 * np.pi / length * np.arange(n // 2 + 1)).reshape(sh)
    F = np.fft.rfft(f, axis=axis)
    if order == 1:
        k = np.where(np.arange(n // 2 + 1).reshape(sh) < n // 2, k, 0.0)
        return np.fft.irfft(1j * k * F, n=n, axis=axis)
    return np.fft.irfft(-k * k * F, n=n, axis=axis)


def _close(got, want, f, axis, order, what):
    n = f.shape[axis]
    kmax = (np.pi * n / 4.0) ** order
    # the pairs of lines share an exponent: the norm of the whole plane bounds both
    tol = 10 * EPS * (1 + np.log2(n)) * kmax * np.abs(f).max(axis=(1, 2), keepdims=True) * np.sqrt(2.0)
    assert (np.abs(got - want) <= tol).all(), (what, n, float((np.abs(got - want) / np.maximum(tol, 1e-300)).max()))


@pytest.mark.parametrize("n", [4, 6, 8, 10, 16, 18, 30, 32, 48, 54, 60, 64, 90, 96, 100, 128, 150, 192, 250, 256, 360, 384,
                               480, 512, 768, 1000, 1024, 1500, 1536, 2000, 2048])
def test_lengths(n):
    rng = np.random.default_rng(n)
    for nx, ny, axis in ((n, 18, 2), (18, n, 1)):
        f = rng.standard_normal((6, ny, nx))
        f[1] += 100.0                                     # a constant plus little
        f[2] = np.cos(2 * np.pi * np.arange(n) / n).reshape((-1, 1) if axis == 1 else (1, -1)) + 0 * f[2]
        f[3] = 0.0
        f[4] = 0.0
        f[4, 2, 3] = 7.0                                  # a spike
        f[5] *= 10.0 ** rng.uniform(-8, 8, (ny, 1) if axis == 2 else (1, nx))
        g = P3D(convection_params(nx, ny, 6))
        a, b = g.d2bydx(f) if axis == 2 else g.d2bydy(f)
        c = g.d1bydx(f) if axis == 2 else g.d1bydy(f)
        assert np.array_equal(a, c)
        _close(a, _ref(f, axis, 1), f, axis, 1, "d1")
        _close(b, _ref(f, axis, 2), f, axis, 2, "d2")
        h = g.inversefft(g.forwardfft(f))
        _close(h, f, f, axis, 0, "round trip")
        g.close()


@pytest.mark.parametrize("scale", [1e-320, 1e-300, 1e-155, 1e155, 1e290])
def test_scales(scale):
    """The operators are linear up to the rounding of the subnormal range."""
    rng = np.random.default_rng(5)
    f = rng.standard_normal((6, 12, 60))
    g = P3D(convection_params(60, 12, 6))
    s = f * scale
    want = g.d1bydx(s / scale if scale > 1e-310 else f) * scale
    got = g.d1bydx(s)
    # subnormal inputs and outputs are multiples of 2^-1074
    tol = 1e-12 * np.abs(want).max() + (200 * 2.0 ** -1074 if scale < 1e-290 else 0.0)
    assert np.isfinite(got).all() and np.abs(got - want).max() <= tol
    g.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_lines(bad):
    """A NaN or infinity spoils its pair of lines and no other."""
    rng = np.random.default_rng(6)
    f = rng.standard_normal((6, 10, 64))
    g = P3D(convection_params(64, 10, 6))
    clean = g.d1bydx(f)
    f[2, 5, 17] = bad
    got = g.d1bydx(f)
    assert np.isnan(got[2, 4:6]).all()
    got[2, 4:6] = clean[2, 4:6]
    assert np.array_equal(got, clean)
    g.close()
