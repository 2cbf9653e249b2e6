"""The ensemble's tuner: where every bound of the z chunk gives the same chunk (grids that
the bound's chunks would not fill the device with, the FP64 form) there is nothing to
choose, and the default stays; where they differ, any of them may win."""
import pytest

from fug30v0kxc_gb300.params import VEC_PREC_FP64, VEC_PREC_SPLIT, convection_params
from fug30v0kxc_gb300.solver import Ensemble

pytestmark = pytest.mark.gpu


def _tuned(shapes, prec):
    ps = [convection_params(*s, ra=1e5, q=100.0, eta_contrast=5.0, precision=prec) for s in shapes]
    e = Ensemble(ps)
    e.start()
    e.tune(steps=1)
    kc = [m.tunables()[0] for m in e.members]
    assert e.step(2) == 0
    e.sync()
    e.close()
    return kc


def test_nothing_to_choose():
    small = [(64, 64, 65), (64, 32, 65), (32, 32, 33), (64, 64, 33), (32, 64, 49)]
    assert _tuned(small, VEC_PREC_SPLIT) == [16] * 5
    assert _tuned([(32, 32, 17), (48, 32, 17), (32, 48, 17)], VEC_PREC_FP64) == [16] * 3


def test_something_to_choose():
    assert set(_tuned([(256, 256, 65)], VEC_PREC_SPLIT)) <= {8, 16, 32}
    # nine members of one grid: their launch takes the bound's own chunks
    kc = _tuned([(64, 64, 65)] * 9, VEC_PREC_SPLIT)
    assert len(set(kc)) == 1 and kc[0] in (8, 16, 32)
