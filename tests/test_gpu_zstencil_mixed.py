"""FP64 right-hand sides beside a spike: several z stencils of a field share their
alignment, and one must not lose bits to a plane that it does not read.

With w > 0 the stencils at plane k read k - 3 .. k + 2 (the upwind one) and k - 2 .. k + 2:
a spike at plane ks = k + 3 is read by none, and the right-hand sides at k are those of the
state without it up to the rounding of the sums, which is the same sum's of the same values
(bound: 64 units in the last place of a largest term, over a thousand terms).  (dw/dt holds
d/dz of dw/dz, which does reach the spike of w.)"""
import numpy as np
import pytest

from helpers import smooth_state
from fug30v0kxc_gb300.params import VEC_PREC_FP64, convection_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field", ["t", "u", "v", "w", "r"])
@pytest.mark.parametrize("size", [1e6, 1e12, 1e200])
def test_spike_out_of_reach(field, size):
    p = convection_params(16, 12, 24, q=0.0, precision=VEC_PREC_FP64)
    s = smooth_state(p, seed=3)
    s["w"] = np.abs(s["w"]) + 0.1
    ks, out = 13, []
    g = P3D(p)
    for spike in (False, True):
        for n in ("r", "t", "u", "v", "w"):
            a = s[n].copy()
            if spike and n == field:
                a[ks] = size
            g.set(n, a)
        g.hydro_deriv()
        out.append({n: g.get(n)[ks - 3] for n in ("rdot3", "tdot3", "udot3", "vdot3", "wdot3")})
    for n, a in out[0].items():
        if field == "w" and n == "wdot3":
            continue
        tol = 64 * 1000 * 2.0 ** -52 * max(1.0, np.abs(a).max())
        assert np.abs(out[1][n] - a).max() <= tol, (n, float(np.abs(out[1][n] - a).max() / tol))
    g.close()
