"""FP64 contexts with more planes than a grid has rows (65535): the z operators, the
hydro right-hand sides, calcdt and a step.

The operators against their own stencils in long double on interior planes (bound: that
of the z stencil tests), the right-hand sides of a state that repeats every 40 planes by
planes 40 apart: away from the walls they have equal bits."""
import ctypes as C
import time

import numpy as np
import pytest

from fug30v0kxc_gb300.params import VEC_PREC_FP64, convection_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(4, 4, 65536), (4, 6, 70000), (16, 20, 65535)])
def test_operators(nx, ny, nz):
    rng = np.random.default_rng(nz)
    g = P3D(convection_params(nx, ny, nz))
    f = rng.standard_normal((nz, ny, nx))
    h = (nz - 1) / 12.0
    x = f.astype(np.longdouble)
    d1 = h * (x[:-4] - 8 * x[1:-3] + 8 * x[3:-1] - x[4:])
    top = np.abs(f).max()
    assert np.abs(g.d1bydz(f, 5)[2:-2] - d1).max() <= h * 80 * 2.0 ** -52 * top
    g.set("w", np.ones_like(f))
    up = h * (-x[:-5] + 6 * x[1:-4] - 18 * x[2:-3] + 10 * x[3:-2] + 3 * x[4:-1])
    assert np.abs(g.d1upbydz(f, 5)[3:-2] - up).max() <= h * 80 * 2.0 ** -52 * top
    g.close()


@pytest.mark.parametrize("nz", [65536, 70000])
def test_step(nz):
    p = convection_params(4, 4, nz, q=0.0, precision=VEC_PREC_FP64)
    g = P3D(p)
    rng = np.random.default_rng(1)
    rep = lambda a: np.tile(a, (nz // 40 + 1, 1, 1))[:nz]     # noqa: E731
    for n, c in (("r", 1.0), ("t", 1.0), ("u", 0.0), ("v", 0.0), ("w", 0.0)):
        g.set(n, rep(c + 1e-3 * rng.standard_normal((40, 4, 4))))
    g.hydro_deriv()
    for n in ("rdot3", "udot3", "vdot3", "wdot3"):
        a = g.get(n)
        assert np.isfinite(a).all() and np.array_equal(a[8:-48], a[48:-8]), n
    dt = g.calcdt()
    assert np.isfinite(dt) and dt > 0.0
    assert g.step(1) == 0
    g.close()


@pytest.mark.parametrize("nz", [46341, 46342, 70000])
def test_second_derivative(nz):
    """(nz - 1)^2 does not fit 32 bits above 46341 planes."""
    g = P3D(convection_params(4, 4, nz))
    f = np.random.default_rng(nz).standard_normal((nz, 4, 4))
    s, x = (nz - 1) ** 2 / 12.0, f.astype(np.longdouble)
    d2 = s * (-x[:-4] + 16 * x[1:-3] - 30 * x[2:-2] + 16 * x[3:-1] - x[4:])
    assert np.abs(g.d2bydz(f, 3)[2:-2] - d2).max() <= s * 700 * 2.0 ** -52 * np.abs(f).max()
    g.close()


def test_columns_fill_their_blocks():
    """A column of 60000 values takes a call's fixed time, as one of 1000 does (with a CTA per
    value it took three times as long)."""
    torch = pytest.importorskip("torch")
    ts = []
    for nz in (1000, 60000):
        g = P3D(convection_params(4, 4, nz))
        f = torch.randn(nz, dtype=torch.float64, device="cuda")
        o = torch.empty_like(f)
        t = []
        for _ in range(100):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            assert g.L.vec_d1bydz1d(g.h, C.c_void_p(f.data_ptr()), C.c_void_p(o.data_ptr()), 5) == 0
            t.append(time.perf_counter() - t0)
        ts.append(sorted(t)[25])
        g.close()
    assert ts[1] <= 1.8 * ts[0], ts
