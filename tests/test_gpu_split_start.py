"""The start of a split run (mag_init's FP64 transforms of B) where both lengths are the
register kernel's, where only one is, and where none is, against the FP64 form's."""
import numpy as np
import pytest

from fug30v0kxc_gb300.params import VEC_PREC_SPLIT, convection_params
from fug30v0kxc_gb300.solver import P3D
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(64, 64), (96, 64), (128, 192), (256, 96), (60, 64), (64, 50), (30, 54), (384, 64)])
def test_mag_init(nx, ny):
    got = []
    for split in (False, True):
        p = convection_params(nx, ny, 9, eta_contrast=5.0)
        if split:
            p.precision = VEC_PREC_SPLIT
        g = P3D(p)
        g.start()
        rng = np.random.default_rng(nx * ny)
        for n in ("bx", "by", "bz"):
            g.set(n, rng.standard_normal((9, ny, nx)))
        g.mag_init()
        got.append({n: g.get(n) for n in ("pol", "tor")})
        g.close()
    # two FP64 transforms: rounding of a few 1e-16 times log2 of the plane's size
    for n in ("pol", "tor"):
        assert rel_err(got[1][n], got[0][n]) < 1e-13, n
