"""The error of the FP32 line operators against FP64, on lines of few waves, the same with
a little noise, a constant plus little, and white noise.

BOUND holds the root-mean-square errors, relative to the result's, that this library's
plain two-level transforms (register kernel and Stockham passes, one line pair per group)
have on these lines: derivatives of smooth lines weigh what a transform rounds off at high
wavenumbers, which the order of its radices and its twiddles decide.  A kernel may not err
more; 1 % for the spread between samples of lines (2 % for the lengths of the general
kernel, which divides its multiply-adds otherwise)."""
import ctypes as C

import numpy as np
import pytest

from fug30v0kxc_gb300.params import convection_params
from fug30v0kxc_gb300.solver import P3D

pytestmark = pytest.mark.gpu
KINDS = ("waves", "noisy", "constant", "white")
# (d1, d2, dealias)
BOUND = {
    30: {"waves": (4.094e-07, 2.532e-06, 1.028e-07),
         "noisy": (4.309e-07, 2.297e-06, 1.095e-07),
         "constant": (1.744e-04, 1.057e-03, 8.451e-08),
         "white": (1.180e-07, 1.119e-07, 1.226e-07)},
    60: {"waves": (3.330e-07, 1.528e-06, 1.144e-07),
         "noisy": (3.496e-07, 1.532e-06, 1.191e-07),
         "constant": (1.359e-04, 6.262e-04, 9.116e-08),
         "white": (1.238e-07, 1.218e-07, 1.308e-07)},
    90: {"waves": (3.597e-07, 1.496e-06, 1.142e-07),
         "noisy": (3.651e-07, 1.466e-06, 1.188e-07),
         "constant": (1.491e-04, 6.257e-04, 8.149e-08),
         "white": (1.366e-07, 1.352e-07, 1.316e-07)},
    240: {"waves": (3.723e-07, 1.453e-06, 1.222e-07),
          "noisy": (3.813e-07, 1.453e-06, 1.290e-07),
          "constant": (1.260e-04, 5.176e-04, 9.562e-08),
          "white": (1.493e-07, 1.484e-07, 1.409e-07)},
    320: {"waves": (3.732e-07, 1.445e-06, 1.208e-07),
          "noisy": (3.770e-07, 1.424e-06, 1.278e-07),
          "constant": (1.209e-04, 5.046e-04, 8.111e-08),
          "white": (1.473e-07, 1.472e-07, 1.399e-07)},
    360: {"waves": (3.831e-07, 1.474e-06, 1.253e-07),
          "noisy": (3.926e-07, 1.477e-06, 1.323e-07),
          "constant": (1.402e-04, 5.577e-04, 8.553e-08),
          "white": (1.517e-07, 1.516e-07, 1.456e-07)},
    384: {"waves": (3.872e-07, 1.462e-06, 1.296e-07),
          "noisy": (3.923e-07, 1.450e-06, 1.348e-07),
          "constant": (1.174e-04, 5.002e-04, 7.328e-08),
          "white": (1.659e-07, 1.668e-07, 1.492e-07)},
    480: {"waves": (3.986e-07, 1.533e-06, 1.270e-07),
          "noisy": (4.064e-07, 1.522e-06, 1.349e-07),
          "constant": (1.310e-04, 5.307e-04, 9.536e-08),
          "white": (1.587e-07, 1.586e-07, 1.481e-07)},
    512: {"waves": (4.050e-07, 1.565e-06, 1.378e-07),
          "noisy": (4.113e-07, 1.561e-06, 1.460e-07),
          "constant": (1.186e-04, 5.264e-04, 6.728e-08),
          "white": (1.639e-07, 1.665e-07, 1.581e-07)},
    640: {"waves": (3.974e-07, 1.523e-06, 1.271e-07),
          "noisy": (4.034e-07, 1.512e-06, 1.364e-07),
          "constant": (1.231e-04, 5.051e-04, 8.315e-08),
          "white": (1.562e-07, 1.565e-07, 1.497e-07)},
    768: {"waves": (4.236e-07, 1.606e-06, 1.402e-07),
          "noisy": (4.271e-07, 1.581e-06, 1.475e-07),
          "constant": (1.255e-04, 5.193e-04, 7.402e-08),
          "white": (1.785e-07, 1.796e-07, 1.616e-07)},
    1000: {"waves": (4.341e-07, 1.662e-06, 1.709e-07),
           "noisy": (4.445e-07, 1.664e-06, 1.779e-07),
           "constant": (1.536e-04, 6.062e-04, 1.000e-07),
           "white": (1.743e-07, 1.755e-07, 1.908e-07)},
    1024: {"waves": (4.317e-07, 1.665e-06, 1.480e-07),
           "noisy": (4.372e-07, 1.657e-06, 1.564e-07),
           "constant": (1.247e-04, 5.455e-04, 6.933e-08),
           "white": (1.753e-07, 1.765e-07, 1.707e-07)},
    1280: {"waves": (4.172e-07, 1.594e-06, 1.321e-07),
           "noisy": (4.174e-07, 1.555e-06, 1.421e-07),
           "constant": (1.266e-04, 5.125e-04, 8.440e-08),
           "white": (1.624e-07, 1.628e-07, 1.565e-07)},
    1500: {"waves": (4.484e-07, 1.726e-06, 1.460e-07),
           "noisy": (4.587e-07, 1.723e-06, 1.556e-07),
           "constant": (1.668e-04, 6.614e-04, 9.275e-08),
           "white": (1.763e-07, 1.755e-07, 1.699e-07)},
    2048: {"waves": (4.395e-07, 1.705e-06, 1.377e-07),
           "noisy": (4.439e-07, 1.690e-06, 1.483e-07),
           "constant": (1.252e-04, 5.300e-04, 6.870e-08),
           "white": (1.689e-07, 1.695e-07, 1.633e-07)},
}


def lines(n, kind, m):
    rng = np.random.default_rng(n + 1)
    x = np.arange(n) / n
    if kind == "white":
        return (2 * rng.random((m, n)) - 1).astype(np.float32)
    f = np.zeros((m, n))
    for _ in range(4):
        k = rng.integers(0, max(2, n // 8), (m, 1))
        f += (rng.random((m, 1)) - 0.5) * np.cos(2 * np.pi * (k * x + rng.random((m, 1))))
    if kind == "noisy":
        f += 1e-2 * (2 * rng.random((m, n)) - 1)
    elif kind == "constant":
        f = 1 + 3 * rng.random((m, 1)) + 1e-2 * f
    return f.astype(np.float32)


def errors(n, kind, dim, m=256, nz=12):
    """rms errors of d1, d2 and dealias along x (dim 0) or y."""
    torch = pytest.importorskip("torch")
    f = lines(n, kind, m * nz)
    k = np.pi / 2 * np.arange(n // 2 + 1)
    k1 = np.where(np.arange(n // 2 + 1) < n // 2, k, 0.0)
    F = np.fft.rfft(f.astype(np.float64), axis=1)
    keep = np.arange(n // 2 + 1) < n // 2 - (n // 2) // 3
    want = [np.fft.irfft(s * F, n=n, axis=1) for s in (1j * k1, -k * k, keep)]
    g = P3D(convection_params(*((n, m) if dim == 0 else (m, n)), nz))
    a = f.reshape(nz, m, n)
    t = torch.tensor(np.ascontiguousarray(a if dim == 0 else a.transpose(0, 2, 1)), device="cuda")
    o = [torch.empty_like(t) for _ in range(3)]
    p = [C.c_void_p(q.data_ptr()) for q in [t] + o]
    torch.cuda.synchronize()
    assert g.L.vec_line_f32(g.h, dim, 1, 2, p[0], p[1], p[2]) == 0
    assert g.L.vec_line_f32(g.h, dim, 3, 0, p[0], p[3], None) == 0
    got = [q.cpu().numpy() for q in o]
    g.close()
    got = [(q if dim == 0 else q.transpose(0, 2, 1)).reshape(m * nz, n) for q in got]
    return [float(np.sqrt(((q - w) ** 2).mean() / (w * w).mean())) for q, w in zip(got, want)]


@pytest.mark.parametrize("dim", [0, 1])
@pytest.mark.parametrize("n", sorted(BOUND))
def test_error(n, dim):
    for kind in KINDS:
        e = errors(n, kind, dim)
        slack = 1.01 if n in (384, 512, 768, 1024) else 1.02
        assert all(a <= slack * b for a, b in zip(e, BOUND[n][kind])), (kind, e, BOUND[n][kind])
