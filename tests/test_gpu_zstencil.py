"""The FP64 z stencils (sums in integers inside, FP64 at the walls and where the
values leave the integers' range) against the oracle and against numpy in long
double, on fields whose planes differ by many orders of magnitude, with zeros,
infinities and values near both ends of the exponent range.

The integer sum keeps three bits below the last one of the largest neighbour:
its error is at most one unit of those per neighbour and weight (64 in all, 8
units in the last place) and one rounding."""
import numpy as np
import pytest

from oracle import oracle as O
from fug30v0kxc_gb300.params import default_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu


def _pair(nx, ny, nz):
    p = default_params()
    p.nx, p.ny, p.nz = nx, ny, nz
    return P3D(p), O.Oracle(p)


def _bound(f, weights):
    """Largest neighbour within three planes, times the tolerance."""
    a = np.abs(f)
    m = a.copy()
    for d in range(1, 6):
        m[d:] = np.maximum(m[d:], a[:-d])
        m[:-d] = np.maximum(m[:-d], a[d:])
    return m * (weights * 2.0 ** -52)


@pytest.mark.parametrize("nz", [6, 7, 8, 33])
@pytest.mark.parametrize("kind", ["plain", "planes", "points", "tiny", "huge", "zeros", "walls"])
def test_stencils(nz, kind):
    nx, ny = 12, 6
    g, o = _pair(nx, ny, nz)
    rng = np.random.default_rng(nz)
    f = rng.standard_normal((nz, ny, nx))
    if kind == "planes":
        f *= 10.0 ** rng.uniform(-12, 12, (nz, 1, 1))
    elif kind == "points":
        f *= 10.0 ** rng.uniform(-30, 30, f.shape)
    elif kind == "tiny":
        f *= 1e-300
    elif kind == "huge":
        f *= 1e300
    elif kind == "zeros":
        f[rng.random(f.shape) < 0.7] = 0.0
    elif kind == "walls":
        f = np.sin(np.pi * np.arange(nz) / (nz - 1))[:, None, None] ** 3 * f
    w = rng.standard_normal(f.shape)
    g.set("w", w)
    o.set("w", w)
    h, s = (nz - 1) / 12.0, (nz - 1) ** 2 / 12.0
    for fl in (0, 1, 2, 5):
        assert (np.abs(g.d1bydz(f, fl) - o.d1bydz(f, fl)) <= h * _bound(f, 80)).all(), (kind, fl)
        assert (np.abs(g.d1upbydz(f, fl) - o.d1upbydz(f, fl)) <= h * _bound(f, 80)).all(), (kind, fl)
    for fl in (0, 3):
        assert (np.abs(g.d2bydz(f, fl) - o.d2bydz(f, fl)) <= s * _bound(f, 700)).all(), (kind, fl)
    # integers on the interior rows: exact
    f = rng.integers(-1000, 1000, f.shape).astype(float)
    d = g.d1bydz(f, 0)
    if nz > 7:
        want = h * (f[1:-6] - 8 * f[2:-5] + 8 * f[4:-3] - f[5:-2])
        assert np.array_equal(d[3:-3][:want.shape[0]], want)
    g.close()
    o.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite(bad):
    g, _ = _pair(12, 6, 20)
    f = np.random.default_rng(1).standard_normal((20, 6, 12))
    clean = g.d1bydz(f, 5)
    f[10, 3, 4] = bad
    got = g.d1bydz(f, 5)
    for k in (8, 9, 11, 12):
        assert not np.isfinite(got[k, 3, 4])
        got[k, 3, 4] = clean[k, 3, 4]
    assert np.array_equal(got, clean)
    g.close()
