"""The split form's dealias step where its pairs of points leave a partial CTA, against
the FP64 form: the same truncation of the same perturbation, at FP32 accuracy."""
import numpy as np
import pytest

from fug30v0kxc_gb300.params import VEC_PREC_SPLIT, convection_params
from fug30v0kxc_gb300.solver import P3D
from tests.test_gpu_split import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(10, 18, 6), (30, 30, 9), (64, 50, 17), (96, 48, 12)])
def test_dealias_step(nx, ny, nz):
    got = []
    for prec in (None, VEC_PREC_SPLIT):
        p = convection_params(nx, ny, nz, eta_contrast=5.0)
        if prec is not None:
            p.precision = prec
        p.ndu06 = 1000
        g = P3D(p)
        g.start()
        assert g.step(11) == 0
        got.append({n: g.get(n) for n in ("r", "t", "u", "v", "w")})
        g.close()
    z = np.arange(nz) / (nz - 1)
    t0 = (1.0 + p.theta * z)[:, None, None]
    for n, bgd in (("r", t0 ** p.cm), ("t", t0), ("u", 0.0), ("v", 0.0), ("w", 0.0)):
        # (1e-4: the bound of the split form's other comparisons with FP64)
        assert rel_l2(got[1][n] - bgd, got[0][n] - bgd) < 1e-4, n
