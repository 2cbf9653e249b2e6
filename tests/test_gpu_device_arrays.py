"""Operators on device arrays: the kernels work on the caller's arrays where
these are aligned and do not overlap, and through the context's scratch
otherwise.  Every form has to give the bits that host arrays give."""
import ctypes as C

import numpy as np
import pytest

from fug30v0kxc_gb300.params import FIELD_NAMES, VEC_PREC_FP64, VEC_PREC_SPLIT, convection_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu


def _arrays(torch, n, off, dtype):
    """n-element views at `off` elements from a 256-byte boundary, apart."""
    big = [torch.zeros(n + 64, dtype=dtype, device="cuda") for _ in range(3)]
    return [b[off:off + n] for b in big]


@pytest.mark.parametrize("nx,ny,nz", [(64, 32, 7), (30, 20, 9), (96, 10, 6)])
@pytest.mark.parametrize("off", [0, 2, 1])
def test_device_matches_host(nx, ny, nz, off):
    torch = pytest.importorskip("torch")
    g = P3D(convection_params(nx, ny, nz))
    rng = np.random.default_rng(nx)
    f = rng.standard_normal((nz, ny, nx))
    n, L, h = f.size, g.L, g.h
    g.set("w", rng.standard_normal(f.shape))

    def dev(x, a):
        a.copy_(torch.from_numpy(np.ascontiguousarray(x)).reshape(-1))
        torch.cuda.synchronize()
        return C.c_void_p(a.data_ptr())

    def same(a, want):
        assert np.array_equal(a.cpu().numpy().reshape(want.shape), want)

    a, b, c = _arrays(torch, n, off, torch.float64)
    pb, pc = C.c_void_p(b.data_ptr()), C.c_void_p(c.data_ptr())
    pa = dev(f, a)
    for fn, host in ((L.vec_d2bydx, g.d2bydx), (L.vec_d2bydy, g.d2bydy)):
        assert fn(h, pa, pb, pc) == 0
        for x, y in zip((b, c), host(f)):
            same(x, y)
    for fn, host in ((L.vec_d1bydx, g.d1bydx), (L.vec_d1bydy, g.d1bydy), (L.vec_forwardfft, g.forwardfft),
                     (L.vec_inversefft, g.inversefft)):
        pa = dev(f, a)
        assert fn(h, pa, pb) == 0
        want = host(f)
        same(b, want)
        assert fn(h, pa, pa) == 0          # in place
        same(a, want)
    pa = dev(f, a)
    assert L.vec_dealias(h, pa) == 0
    same(a, g.dealias(f))
    for fn, host, fl in ((L.vec_d1bydz, g.d1bydz, 5), (L.vec_d1upbydz, g.d1upbydz, 1), (L.vec_d2bydz, g.d2bydz, 3)):
        pa = dev(f, a)
        assert fn(h, pa, pb, fl) == 0
        want = host(f, fl)
        same(b, want)
        assert fn(h, pa, pa, fl) == 0      # in place: through the scratch
        same(a, want)
    # an output that starts inside the input
    big = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
    pa = dev(f, big[:n])
    assert L.vec_d1bydx(h, pa, C.c_void_p(big.data_ptr() + 8 * (nx * ny))) == 0
    same(big[nx * ny:nx * ny + n], g.d1bydx(f))
    # FP32 lines, both outputs
    f32 = f.astype(np.float32)
    a, b, c = _arrays(torch, n, 2 * off, torch.float32)
    for d in (0, 1):
        pa = dev(f32, a)
        assert L.vec_line_f32(h, d, 1, 2, pa, C.c_void_p(b.data_ptr()), C.c_void_p(c.data_ptr())) == 0
        for x, y in zip((b, c), g.line_f32(d, 1, f32, 2)):
            same(x, y)
    g.close()


@pytest.mark.parametrize("precision", [VEC_PREC_FP64, VEC_PREC_SPLIT])
def test_fields_and_histories(precision):
    """set / get of the state and of the right-hand sides by logical slot,
    device and host, through history shifts."""
    torch = pytest.importorskip("torch")
    g = P3D(convection_params(32, 16, 8, precision=precision))
    g.start()
    rng = np.random.default_rng(2)
    for k in range(4):
        assert g.step(1) == 0
        for name in ("rdot1", "udot2", "wdot3", "t", "bx", "tordot3"):
            want = g.get(name)
            d = torch.zeros(want.shape, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            assert g.L.vec_get_field(g.h, FIELD_NAMES[name], C.c_void_p(d.data_ptr())) == 0
            assert np.array_equal(d.cpu().numpy(), want), name
        x = rng.standard_normal(want.shape).astype(np.float32).astype(np.float64)
        keep = g.get("vdot2")
        for src in (x, torch.from_numpy(x).cuda()):
            torch.cuda.synchronize()
            p = src.ctypes.data if isinstance(src, np.ndarray) else src.data_ptr()
            assert g.L.vec_set_field(g.h, FIELD_NAMES["vdot2"], C.c_void_p(p)) == 0
            assert np.array_equal(g.get("vdot2"), x)
        g.set("vdot2", keep)
    g.close()
