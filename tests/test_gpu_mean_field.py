"""The mean field's step inside mag_final's launch against the separate kernels, at
plane counts around the size of its CTA and with all walls in one warp."""
import numpy as np
import pytest

from fug30v0kxc_gb300.params import VEC_PREC_SPLIT, convection_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eta", [1.0, 5.0])
@pytest.mark.parametrize("nz", [6, 9, 32, 33, 255, 256, 257, 300])
def test_mean_field_steps(nz, eta, monkeypatch):
    out = []
    for vec4 in ("1", "0"):
        monkeypatch.setenv("VEC_VEC4", vec4)
        p = convection_params(32, 32, nz, eta_contrast=eta, precision=VEC_PREC_SPLIT)
        p.ndu06 = 10
        g = P3D(p)
        g.start()
        z = np.linspace(0.0, 1.0, nz)
        g.set_mean("bxbar", np.sin(2.0 * z) + z ** 3)
        g.set_mean("bybar", np.cos(3.0 * z))
        assert g.step(4) == 0
        out.append([g.get_mean(m) for m in ("bxbar", "bybar")])
        g.close()
    # the E means come from FP32 sums that the two forms round apart (1e-6 of E, and E
    # enters with dt); the mean's own terms are the same FP64 expressions
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.abs(a - b).max() <= 1e-6 * np.abs(b).max()
