"""FP64 lines of zeros: a field at rest, the truncated rows of a spectrum, and the
missing lines of a partial tile.  They are transformed like any others: exact zeros, a
neighbouring pair of lines with the bits it has beside other lines, and no longer time
than random ones (the bound leaves half as much again for the clock's noise)."""
import ctypes as C
import time

import numpy as np
import pytest

from fug30v0kxc_gb300.params import convection_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 30, 64, 100, 256, 600, 2048])
def test_zeros_beside_others(n):
    rng = np.random.default_rng(n)
    for axis in (2, 1):
        nx, ny = (n, 18) if axis == 2 else (18, n)
        f = rng.standard_normal((6, ny, nx))
        g = P3D(convection_params(nx, ny, 6))
        ops = [lambda a: np.stack(g.d2bydx(a) if axis == 2 else g.d2bydy(a)), g.forwardfft, g.inversefft, g.dealias]
        whole = [op(f) for op in ops]
        z = f.copy()
        lines = np.moveaxis(z, axis, 2)
        lines[1] = 0.0
        lines[2, 4:8] = -0.0                       # two pairs of lines
        lines[3, 4:6] = 5e-324                     # (not zero: the last bit alone)
        got = [op(z) for op in ops]
        first = [np.moveaxis(a, axis - 3, -1) for a in (whole[0], got[0])]
        assert not first[1][:, 1].any() and not first[1][:, 2, 4:8].any()
        keep = np.ones(first[0].shape[1:3], bool)
        keep[1], keep[2, 4:8], keep[3, 4:6] = False, False, False
        assert np.array_equal(first[1][:, keep], first[0][:, keep])
        for a, b in zip(got[1:], whole[1:]):       # (two-dimensional: planes)
            assert not a[1].any()
            for k in (0, 4, 5):
                assert np.array_equal(a[k], b[k])
            assert np.isfinite(a).all()
        g.close()


@pytest.mark.parametrize("nx,ny,nz", [(256, 256, 65), (64, 64, 65), (240, 250, 65)])
def test_zeros_take_no_longer(nx, ny, nz):
    torch = pytest.importorskip("torch")
    g = P3D(convection_params(nx, ny, nz))
    f = torch.randn(nz, ny, nx, dtype=torch.float64, device="cuda")
    rows = f.clone()
    rows[:, : ny // 3] = 0.0
    o = [torch.empty_like(f) for _ in range(2)]
    ptr = [C.c_void_p(a.data_ptr()) for a in o]

    def us(call):
        t = []
        for _ in range(40):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            assert call() == 0
            t.append(time.perf_counter() - t0)
        return sorted(t)[10] * 1e6

    for name in ("d2bydx", "d2bydy", "inversefft"):
        fn = getattr(g.L, "vec_" + name)
        ts = [us(lambda: fn(g.h, C.c_void_p(a.data_ptr()), *(ptr if name != "inversefft" else ptr[:1])))
              for a in (f, torch.zeros_like(f), rows)]
        assert max(ts[1:]) <= 1.5 * ts[0], (name, ts)
    g.close()
