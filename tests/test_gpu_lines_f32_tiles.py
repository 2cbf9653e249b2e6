"""The FP32 register line kernel over several tiles per CTA (both tile buffers, their
reuse, the last partial round), against transforms in double; and its warp- and
group-local barriers against CTA-wide ones, which compute the same."""
import numpy as np
import pytest
import torch

from fug30v0kxc_gb300.params import convection_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu
D1, D2, FWD, INV = 1, 2, 4, 5


def _wavenumbers(n, axis, length):
    k = torch.fft.rfftfreq(n, length / n, dtype=torch.float64, device="cuda") * (2 * np.pi)
    return k.reshape([-1 if q == axis else 1 for q in range(3)])


@pytest.mark.parametrize("n", [64, 96, 128, 192, 256, 384, 512, 768, 1024])
@pytest.mark.parametrize("direction", [0, 1])
def test_many_tiles(n, direction, monkeypatch):
    # at most eight CTAs per SM, two or four tiles per plane
    nz = 1500 if n <= 128 else 500
    nx, ny, axis = (n, 64, 2) if direction == 0 else (64, n, 1)
    f = torch.randn(nz, ny, nx, generator=torch.Generator().manual_seed(n)).numpy()
    p = convection_params(nx, ny, nz)
    g = P3D(p)
    d1, d2 = g.line_f32(direction, D1, f, D2)
    h = g.line_f32(direction, FWD, f)
    back, dback = g.line_f32(direction, INV, h, D1)
    g.close()
    x = torch.from_numpy(f).cuda().double()
    F = torch.fft.rfft(x, dim=axis)
    k = _wavenumbers(n, axis, p.xmax if direction == 0 else p.ymax)
    F1 = F * (1j * k)
    F1.narrow(axis, n // 2, 1).zero_()
    w1 = torch.fft.irfft(F1, n=n, dim=axis)
    w2 = torch.fft.irfft(F * (-k * k), n=n, dim=axis)
    # FP32 rounding of a transform grows like log2(n), below 2^-23 times the largest
    # value per level and product: 1e-5 of it at 1024 points
    for got, want in ((d1, w1), (d2, w2), (back, x), (dback, w1)):
        assert float((torch.from_numpy(got).cuda() - want).abs().max() / want.abs().max()) < 1e-5
    monkeypatch.setenv("VEC_CT_WARP", "0")
    g = P3D(convection_params(nx, ny, nz))
    e1, e2 = g.line_f32(direction, D1, f, D2)
    hh = g.line_f32(direction, FWD, f)
    assert np.array_equal(d1, e1) and np.array_equal(d2, e2) and np.array_equal(h, hh)
    g.close()
