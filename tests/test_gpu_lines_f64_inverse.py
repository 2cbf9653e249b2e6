"""The inverse FP64 x transform with its derivative (bandj): the spectrum's constant
is no part of the derivative and must not cost it bits, and a constant that is not
finite still spoils its pair of lines."""
import numpy as np
import pytest

from fug30v0kxc_gb300.params import VEC_PREC_FP64, convection_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(32, 32), (60, 32), (300, 16), (32, 300)])
def test_derivative_beside_a_large_constant(nx, ny):
    """bz of one wave along y, 10^8 times as strong at kx = 0 as at kx = 3: on the
    row y = 0 d(bz)/dy vanishes and jsq is (d(bz)/dx)^2 of the weak part.

    Bound: twice (a square) the FP64 line tests' 10 eps (1 + log2 n) sqrt(2); the
    10^8 times that of d(bz)/dy, whose wave is a sixtieth of the weak one's derivative,
    enters squared, below it."""
    nz, weak, strong = 16, 1.0, 1.0e8
    p = convection_params(nx, ny, nz, q=100.0, precision=VEC_PREC_FP64)
    g = P3D(p)
    pol = np.zeros(g.shape)
    pol[:, 1, 0], pol[:, 1, 3] = strong, weak
    g.set("pol", pol)
    g.set("tor", np.zeros(g.shape))
    g.bandj()
    j = g.get("jsq")[5:-5, 0]
    kx, ky, x = 2 * np.pi / p.xmax, 2 * np.pi / p.ymax, np.arange(nx) / nx
    d = 2.0 / (nx * ny) * weak * ((3 * kx) ** 2 + ky ** 2) * 2 * 3 * kx * np.sin(2 * np.pi * 3 * x)
    tol = 2 * 10 * 2.0 ** -52 * (1 + np.log2(max(nx, ny))) * np.sqrt(2.0)
    assert np.abs(j - d * d).max() <= tol * (d * d).max(), float(np.abs(j - d * d).max() / (d * d).max() / tol)
    g.close()


@pytest.mark.parametrize("n", [64, 300])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_constant(n, bad):
    f = np.random.default_rng(n).standard_normal((6, 10, n))
    g = P3D(convection_params(n, 10, 6))
    h = g.forwardfft(f)
    clean = g.inversefft(h)
    h[2, 4, 0] = bad                          # of the x line (plane 2, row 4)
    got = g.inversefft(h)
    assert np.isnan(got[2]).all()
    got[2] = clean[2]
    assert np.array_equal(got, clean)
    g.close()
