"""FP64 line derivatives of a large constant plus little at the longest lines.

The line's mean is taken off before its exponent is chosen, so the error is that
of the little alone: the bound of the other FP64 line tests (ten times numpy's own,
eps log2(n) of the norm times the largest multiplier) on the line without its
constant, against numpy's transform in long double.  What is left of the mean is
2^-20 of it, a fiftieth of the waves here."""
import numpy as np
import pytest

from fug30v0kxc_gb300.params import convection_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu
PI = np.longdouble("3.14159265358979323846264338327950288")


@pytest.mark.parametrize("n", [1000, 1024, 1080, 1500, 1536, 2000, 2048])
@pytest.mark.parametrize("const", [1.9, 1.0, -1.5])
def test_constant_plus_little(n, const):
    rng = np.random.default_rng(n)
    m, nz = 4, 6
    x = np.arange(n) / n
    little = sum((rng.random((nz * m, 1)) - 0.5) * np.cos(2 * np.pi * (rng.integers(1, n // 8, (nz * m, 1)) * x + rng.random((nz * m, 1))))
                 for _ in range(4))
    f = const + 1e-4 * little
    F = np.fft.rfft((f.astype(np.longdouble) - np.longdouble(const)), axis=1)
    k = PI / 2 * np.arange(n // 2 + 1).astype(np.longdouble)
    k1 = np.where(np.arange(n // 2 + 1) < n // 2, k, 0)
    want = np.fft.irfft(1j * k1 * F, n=n, axis=1), np.fft.irfft(-k * k * F, n=n, axis=1)
    size = np.abs(f - const).max() * np.sqrt(2.0)
    for axis in (2, 1):
        g = P3D(convection_params(*((n, m) if axis == 2 else (m, n)), nz))
        a = f.reshape(nz, m, n)
        got = g.d2bydx(a) if axis == 2 else g.d2bydy(np.ascontiguousarray(a.transpose(0, 2, 1)))
        for order, (o, w) in enumerate(zip(got, want), 1):
            o = (o if axis == 2 else o.transpose(0, 2, 1)).reshape(nz * m, n)
            tol = 10 * 2.0 ** -52 * (1 + np.log2(n)) * (np.pi * n / 4.0) ** order * size
            assert np.abs(o - w).max() <= tol, (axis, order, float(np.abs(o - w).max() / tol))
        g.close()
