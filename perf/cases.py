"""The work whose speed is measured: what a user of this library has it do.

Kinds of cases (every array is device memory, as in a program that keeps its
fields on the GPU; each call is an entry point of include/vec.h):

* ops         the reference's operator calls on one field, in FP64: d2bydx,
              d2bydy, d1bydx, d1bydy, d1bydz, d2bydz.
* transforms  forwardfft, inversefft and dealias of one field, in FP64.
* lines       the FP32 line operators (derivative pairs, dealias along x and y).
* rhs         hydro_deriv, mag_deriv and bandj on a loaded state.
* step        ten (fp64: two) iterations of the time loop from a loaded state.
* ensemble    ten iterations of a batch of instances of three grids.
* train       Adam iterations of the closure network on stored pairs.

The split form computes in FP32 on an FP64 state: its fields are returned in
FP32, the precision of what is computed.
"""
import ctypes as C
import math

import numpy as np
import torch

from fug30v0kxc_gb300.closure import Closure
from fug30v0kxc_gb300.params import (FIELD_NAMES, VEC_PREC_FP64, VEC_PREC_SPLIT, convection_params)
from fug30v0kxc_gb300.solver import P3D, Ensemble

STATE = ("r", "t", "u", "v", "w", "bx", "by", "bz", "jsq", "pol", "tor")
RHS = ("rdot3", "tdot3", "udot3", "vdot3", "wdot3")
MAG = ("poldot3", "tordot3")


def listed():
    return [
        # the reference's own default grid (bin/INPUT): a mixed-radix length, small calls
        {"name": "ops_30x30x60", "kind": "ops", "nx": 30, "ny": 30, "nz": 60},
        # the headline grid, operator by operator (a host program that keeps its own loop)
        {"name": "ops_256x256x129", "kind": "ops", "nx": 256, "ny": 256, "nz": 129},
        # 3 2^a lines (the ensemble's largest grid)
        {"name": "transforms_192x192x129", "kind": "transforms", "nx": 192, "ny": 192, "nz": 129},
        # the FP32 operators on their own
        {"name": "lines_512x512x65", "kind": "lines", "nx": 512, "ny": 512, "nz": 65},
        # an uneven grid with lengths outside 2^a: right-hand sides of the drop-in form
        {"name": "rhs_fp64_96x60x33", "kind": "rhs", "nx": 96, "ny": 60, "nz": 33, "prec": "fp64", "q": 100.0, "eta": 5.0},
        # right-hand sides at the closure's coarse grid, split form
        {"name": "rhs_split_128x128x65", "kind": "rhs", "nx": 128, "ny": 128, "nz": 65, "prec": "split", "q": 1000.0, "eta": 20.0},
        # the drop-in time loop at the headline grid
        {"name": "step_fp64_256x256x129", "kind": "step", "nx": 256, "ny": 256, "nz": 129, "prec": "fp64", "q": 100.0, "eta": 20.0},
        # the CPU-runnable reference case: small, bound by launches
        {"name": "step_split_64x64x65", "kind": "step", "nx": 64, "ny": 64, "nz": 65, "prec": "split", "q": 100.0, "eta": 5.0},
        # the headline: split form at 256^2 x 129
        {"name": "step_split_256x256x129", "kind": "step", "nx": 256, "ny": 256, "nz": 129, "prec": "split", "q": 100.0, "eta": 20.0},
        # the closure's fine grid
        {"name": "step_split_512x512x257", "kind": "step", "nx": 512, "ny": 512, "nz": 257, "prec": "split", "q": 1000.0, "eta": 20.0},
        # uneven grids and parameters, magnetic and not, in one captured step
        {"name": "ensemble_3x3", "kind": "ensemble", "per_grid": 3, "nmax": 192},
        # training of the learned closure, batch 8 at its coarse grid
        {"name": "train_128x128x65", "kind": "train", "nx": 128, "ny": 128, "nz": 65},
    ]


def draw(rng):
    """One more case of the same ranges."""
    def log(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    def length(top):
        # lengths 2^a 3^b 5^c that are even, as the solver takes them
        ok = [n for n in range(30, top + 1, 2) if _smooth(n)]
        x = log(30, top)
        return min(ok, key=lambda n: (abs(math.log(n / x)), n))

    kind = rng.choice(["ops", "ops", "transforms", "lines", "rhs", "rhs", "step", "step", "step", "ensemble"])
    top = 512 if rng.random() < 0.25 else 256
    # square grids of the tuned lengths and uneven ones of any length
    if rng.random() < 0.6:
        nx = ny = rng.choice([n for n in (64, 96, 128, 192, 256, 384, 512) if n <= top])
    else:
        nx, ny = length(top), length(top)
    nz = int(round(log(17, 129)))
    prec = rng.choice(["fp64", "split"])
    q, eta = rng.choice([0.0, 100.0, 1000.0]), rng.choice([1.0, 5.0, 20.0])
    if kind == "ensemble":
        return {"kind": kind, "per_grid": rng.randint(1, 3), "nmax": rng.choice([96, 128, 192])}
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    if kind == "rhs" or kind == "step":
        c.update(prec=prec, q=q, eta=eta)
        # the FP64 form costs an order of magnitude more per point
        if prec == "fp64" and nx * ny * nz > 256 * 256 * 129:
            c.update(nx=256, ny=256)
    return c


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


# ---- inputs -----------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _horiz(g, shape, lx=4.0, modes=4):
    """A smooth periodic field of every plane: a few long waves, their
    amplitudes drawn anew per plane, shape (nz, ny, nx)."""
    nz, ny, nx = shape
    d = dict(dtype=torch.float64, device="cuda")
    x, y = torch.arange(nx, **d) / nx, torch.arange(ny, **d) / ny
    z = torch.linspace(0, 1, nz, **d)
    f = torch.zeros(shape, **d)
    for _ in range(modes):
        kx, ky = (int(torch.randint(0, max(2, n // 8), (1,), generator=g, device="cuda")) for n in (nx, ny))
        ph, a, b = torch.rand(3, generator=g, **d).tolist()
        prof = (1 + 0.3 * torch.cos(math.pi * z * (1 + 2 * b)))[:, None, None] * (a - 0.5)
        f += prof * torch.cos(2 * math.pi * (kx * x[None, None, :] + ky * y[None, :, None] + ph))
    return f


def _noise(g, shape):
    return 2 * torch.rand(shape, generator=g, dtype=torch.float64, device="cuda") - 1


def _fields(p, seed, amp=1e-2, bamp=5e-2, noise=1e-4):
    """A convecting layer: the polytrope with waves and grid noise in r, T, u,
    v, w (velocities vanish at the walls) and a disturbed vertical field."""
    g, shape = _gen(seed), (p.nz, p.ny, p.nx)
    z = torch.linspace(0, 1, p.nz, dtype=torch.float64, device="cuda")[:, None, None]
    wall, t0 = torch.sin(math.pi * z), 1.0 + p.theta * z
    s = {n: wall * (amp * _horiz(g, shape) + noise * _noise(g, shape)) for n in ("u", "v", "w", "t", "r")}
    s["t"] = t0 + s["t"]
    s["r"] = t0 ** p.cm * (1.0 + s["r"])
    on = 1.0 if p.f else 0.0
    for n in ("bx", "by"):
        s[n] = on * bamp * torch.cos(math.pi * z) * _horiz(g, shape)
    s["bz"] = on * (1.0 + bamp * _horiz(g, shape))
    return s


def _params(c):
    prec = VEC_PREC_SPLIT if c["prec"] == "split" else VEC_PREC_FP64
    p = convection_params(c["nx"], c["ny"], c["nz"], q=c["q"], eta_contrast=c["eta"], precision=prec)
    p.ndu06 = 1000000
    return p


def _ptr(a):
    return C.c_void_p(a.data_ptr())


def _ok(st, what):
    if st != 0:
        raise RuntimeError("%s: status %d" % (what, st))


def _set(g, fields):
    torch.cuda.synchronize()
    for n, a in fields.items():
        _ok(g.L.vec_set_field(g.h, FIELD_NAMES[n], _ptr(a)), n)


def _get(g, names, out):
    for n in names:
        _ok(g.L.vec_get_field(g.h, FIELD_NAMES[n], _ptr(out[n])), n)


def _buffers(names, shape):
    return {n: torch.zeros(shape, dtype=torch.float64, device="cuda") for n in names}


def _member_params(c):
    grids = [g for g in ((64, 65), (96, 81), (128, 97), (192, 129)) if g[0] <= c["nmax"]][-3:]
    rng, ps = np.random.default_rng(20240), []
    for n, nz in grids:
        for i in range(c["per_grid"]):
            p = convection_params(n, n, nz, ra=float(10.0 ** rng.uniform(4.0, 5.0)), q=(100.0, 0.0, 1000.0)[i % 3],
                                  eta_contrast=(5.0, 1.0, 20.0)[i % 3], precision=VEC_PREC_SPLIT)
            p.ntotal, p.ndu06 = 5000, 1000000
            ps.append(p)
    return ps


def prepare(case, seed):
    k = case["kind"]
    torch.cuda.synchronize()
    if k in ("ops", "transforms", "lines"):
        shape = (case["nz"], case["ny"], case["nx"])
        # (a context of the operators' grid; the operators read no state but w)
        g = P3D(convection_params(case["nx"], case["ny"], case["nz"]))
        gen = _gen(seed)
        f = _horiz(gen, shape) + 1e-2 * _noise(gen, shape)
        dt = torch.float32 if k == "lines" else torch.float64
        n = {"ops": 8, "transforms": 3, "lines": 6}[k]
        return {"case": case, "g": g, "f": f.to(dt), "out": [torch.zeros(shape, dtype=dt, device="cuda") for _ in range(n)]}
    if k in ("rhs", "step"):
        p = _params(case)
        g = P3D(p)
        s = _fields(p, seed)
        if k == "rhs":
            s.update(_spectra(p, seed))
            _set(g, s)
            names = RHS + (MAG + STATE[5:9] if p.f else ())
        else:
            _set(g, s)
            g.calcdt()
            if p.f:
                g.mag_init()
            names = STATE if p.f else STATE[:5]
        return {"case": case, "g": g, "names": names, "out": _buffers(names, g.shape)}
    if k == "ensemble":
        ps = _member_params(case)
        e, outs = Ensemble(ps), []
        for i, (m, p) in enumerate(zip(e.members, ps)):
            _set(m, _fields(p, seed + 1000 * i))
            m.calcdt()
            if p.f:
                m.mag_init()
            outs.append(_buffers(STATE[:7] if p.f else STATE[:5], m.shape))
        return {"case": case, "e": e, "outs": outs}
    # training pairs: a fine run filtered onto a grid half as fine
    fine = P3D(convection_params(2 * case["nx"], 2 * case["ny"], 2 * case["nz"] - 1, ra=1.0e6, q=1.0e3, eta_contrast=20.0,
                                 precision=VEC_PREC_SPLIT))
    pc = convection_params(case["nx"], case["ny"], case["nz"], ra=1.0e6, q=1.0e3, eta_contrast=20.0, precision=VEC_PREC_SPLIT)
    coarse = P3D(pc)
    cl = Closure(pc, factor=2, capacity=8, batch=8, seed=seed)
    _set(fine, _fields(fine.p, seed))
    fine.calcdt()
    fine.mag_init()
    for _ in range(8):
        cl.add_pair(fine, coarse)
        _ok(fine.step(1), "step")
    cl.fit_norm()
    fine.close()
    coarse.close()
    return {"case": case, "cl": cl}


def _spectra(p, seed):
    """Band-limited potentials in the library's halfcomplex layout, and a
    current density: the magnetic state of the right-hand sides."""
    g, shape = _gen(seed + 7), (p.nz, p.ny, p.nx)
    s = {n: 1e-3 * _fwd(_fwd(_horiz(g, shape), 2), 1) for n in ("pol", "tor")}
    s["jsq"] = 0.1 * _horiz(g, shape) ** 2
    return s if p.f else {}


# ---- one pass ---------------------------------------------------------------
def run(state):
    c = state["case"]
    k = c["kind"]
    if k == "ops":
        g, f, o = state["g"], _ptr(state["f"]), state["out"]
        L, h, q = g.L, g.h, [_ptr(x) for x in o]
        _ok(L.vec_d2bydx(h, f, q[0], q[1]), "d2bydx")
        _ok(L.vec_d2bydy(h, f, q[2], q[3]), "d2bydy")
        _ok(L.vec_d1bydx(h, f, q[4]), "d1bydx")
        _ok(L.vec_d1bydy(h, f, q[5]), "d1bydy")
        _ok(L.vec_d1bydz(h, f, q[6], 5), "d1bydz")
        _ok(L.vec_d2bydz(h, f, q[7], 3), "d2bydz")
        return o
    if k == "transforms":
        g, o = state["g"], state["out"]
        L, h, q = g.L, g.h, [_ptr(x) for x in o]
        _ok(L.vec_forwardfft(h, _ptr(state["f"]), q[0]), "forwardfft")
        _ok(L.vec_inversefft(h, q[0], q[1]), "inversefft")
        o[2].copy_(state["f"])
        torch.cuda.current_stream().synchronize()   # the library's stream reads it next
        _ok(L.vec_dealias(h, q[2]), "dealias")
        return o
    if k == "lines":
        g, f, o = state["g"], _ptr(state["f"]), state["out"]
        q = [_ptr(x) for x in o]
        for d in (0, 1):
            _ok(g.L.vec_line_f32(g.h, d, 1, 2, f, q[3 * d], q[3 * d + 1]), "line_f32")
            _ok(g.L.vec_line_f32(g.h, d, 3, 0, f, q[3 * d + 2], None), "line_f32")
        return o
    if k == "rhs":
        g = state["g"]
        g.hydro_deriv()
        if g.p.f:
            g.mag_deriv()
            g.bandj()
        _get(g, state["names"], state["out"])
        return _typed(c["prec"], state["names"], state["out"])
    if k == "step":
        g = state["g"]
        _ok(g.step(10 if c["prec"] == "split" else 2), "step")
        _get(g, state["names"], state["out"])
        return _typed(c["prec"], state["names"], state["out"])
    if k == "ensemble":
        e = state["e"]
        _ok(e.step(10), "ensemble step")
        e.sync()
        got = []
        for m, out in zip(e.members, state["outs"]):
            _get(m, tuple(out), out)
            got.append(_typed("split", tuple(out), out))
        return got
    cl = state["cl"]
    losses = cl.train(2, lr=1e-3, seed=1)
    return {"losses": losses, "params": cl.net.params(), "grads": cl.net.grads()}


def _typed(prec, names, out):
    return [out[n].float() if prec == "split" else out[n] for n in names]


# ---- what a pass cannot do without -------------------------------------------
def work(case):
    k = case["kind"]
    if k == "ensemble":
        return {"bytes": sum(_step_bytes(p.nx * p.ny * p.nz, "split", bool(p.f)) for p in _member_params(case)), "flops": 0}
    n = case["nx"] * case["ny"] * case["nz"]
    if k == "ops":
        return {"bytes": n * 8 * 14, "flops": 0}        # six calls: a field in, one or two out
    if k == "transforms":
        return {"bytes": n * 8 * 6, "flops": 0}
    if k == "lines":
        return {"bytes": n * 4 * 10, "flops": 0}
    if k == "rhs":
        e = 8 if case["prec"] == "fp64" else 4
        return {"bytes": n * e * (5 + 5 + ((2 + 2 + 4 + 2 + 4) if case["q"] else 0)), "flops": 0}
    if k == "step":
        return {"bytes": _step_bytes(n, case["prec"], case["q"] > 0), "flops": 0}
    # forward and two backward products per layer, 27 taps, batch 8, two iterations
    macs = 27 * (9 * 32 + 32 * 32 + 32 * 32 + 32 * 8)
    return {"bytes": n * 8 * 2 * 4 * 17, "flops": 2 * 2 * 3 * macs * n * 8}


def _step_bytes(n, prec, mag):
    """Per step: the FP64 state read and written, the right-hand sides of the
    last two steps read and this step's written."""
    f, steps, e = (7 if mag else 5), (10 if prec == "split" else 2), (4 if prec == "split" else 8)
    return n * steps * f * (16 + 3 * e)


# ---- the same in 64 bits, without the library ---------------------------------
def _hc(F, n, dim):
    """rfft coefficients to the halfcomplex order r0 r1 .. r_n/2 i_(n/2-1) .. i1."""
    im = F.imag.narrow(dim, 1, n // 2 - 1).flip(dim)
    return torch.cat([F.real, im], dim)


def _fwd(f, dim):
    return _hc(torch.fft.rfft(f, dim=dim), f.shape[dim], dim)


def _inv(h, dim):
    n = h.shape[dim]
    im = torch.zeros_like(h.narrow(dim, 0, n // 2 + 1))
    im.narrow(dim, 1, n // 2 - 1).copy_(h.narrow(dim, n // 2 + 1, n // 2 - 1).flip(dim))
    return torch.fft.irfft(torch.complex(h.narrow(dim, 0, n // 2 + 1), im), n=n, dim=dim)


def _k(n, length, dim):
    k = torch.arange(n // 2 + 1, dtype=torch.float64, device="cuda") * (2 * math.pi / length)
    return k.reshape([-1 if d == dim else 1 for d in range(3)])


def _d(f, dim, order, length=4.0):
    n = f.shape[dim]
    k, F = _k(n, length, dim), torch.fft.rfft(f, dim=dim)
    if order == 2:
        return torch.fft.irfft(-k * k * F, n=n, dim=dim)
    k = k * (torch.arange(n // 2 + 1, device="cuda") < n // 2).reshape(k.shape)   # no first derivative at the Nyquist wave
    return torch.fft.irfft(1j * k * F, n=n, dim=dim)


def _dealias(f, dim):
    n = f.shape[dim]
    keep = torch.arange(n // 2 + 1, device="cuda") < n // 2 - (n // 2) // 3
    return torch.fft.irfft(torch.fft.rfft(f, dim=dim) * keep.reshape([-1 if d == dim else 1 for d in range(3)]), n=n, dim=dim)


def _z1(f, flag):
    """Fourth-order d/dz with its wall rows."""
    nz, o = f.shape[0], torch.zeros_like(f)
    o[2:-2] = f[:-4] - 8 * f[1:-3] + 8 * f[3:-1] - f[4:]
    o[1] = -4 * f[0] - 6 * f[1] + 12 * f[2] - 2 * f[3]
    o[-2] = 4 * f[-1] + 6 * f[-2] - 12 * f[-3] + 2 * f[-4]
    if flag in (1, 5):
        a = 14 if flag == 1 else -22
        o[0] = a * f[0] + 36 * f[1] - 18 * f[2] + 4 * f[3]
        o[-1] = -a * f[-1] - 36 * f[-2] + 18 * f[-3] - 4 * f[-4]
    return o * ((nz - 1) / 12.0)


def _zup(f, flag, w):
    """Upwind d/dz: one-sided towards the flow inside, _z1 next to the walls."""
    nz, o = f.shape[0], _z1(f, flag) * (12.0 / (f.shape[0] - 1))
    pos, neg = o.clone(), o.clone()
    pos[3:-2] = -f[:-5] + 6 * f[1:-4] - 18 * f[2:-3] + 10 * f[3:-2] + 3 * f[4:-1]
    pos[2] = 2 * f[0] - 12 * f[1] + 6 * f[2] + 4 * f[3]
    neg[2:-3] = f[5:] - 6 * f[4:-1] + 18 * f[3:-2] - 10 * f[2:-3] - 3 * f[1:-4]
    neg[-3] = -2 * f[-1] + 12 * f[-2] - 6 * f[-3] - 4 * f[-4]
    return torch.where(w >= 0, pos, neg) * ((nz - 1) / 12.0)


def _z2(f, flag):
    nz, o = f.shape[0], torch.zeros_like(f)
    o[2:-2] = -f[:-4] + 16 * f[1:-3] - 30 * f[2:-2] + 16 * f[3:-1] - f[4:]
    o[1] = 10 * f[0] - 15 * f[1] - 4 * f[2] + 14 * f[3] - 6 * f[4] + f[5]
    o[-2] = 10 * f[-1] - 15 * f[-2] - 4 * f[-3] + 14 * f[-4] - 6 * f[-5] + f[-6]
    if flag == 3:
        o[0] = 45 * f[0] - 154 * f[1] + 214 * f[2] - 156 * f[3] + 61 * f[4] - 10 * f[5]
        o[-1] = 45 * f[-1] - 154 * f[-2] + 214 * f[-3] - 156 * f[-4] + 61 * f[-5] - 10 * f[-6]
    return o * ((nz - 1) ** 2 / 12.0)


def _hydro(p, s):
    """Continuity, energy and momentum right-hand sides of the compressible
    layer with conductivity profile kappa(z) and resistivity eta(z)."""
    d = dict(dtype=torch.float64, device="cuda")
    z = torch.linspace(0, 1, p.nz, **d)[:, None, None]
    r, t, u, v, w = (s[n] for n in ("r", "t", "u", "v", "w"))
    b = [s[n] for n in ("bx", "by", "bz")]
    ck, sck, gm = p.ck, p.sigma * p.ck, p.gamma - 1.0
    kap = 0.5 * (torch.tanh(10 * (z - 0.5)) + 1)
    dkap = 5.0 * torch.cosh(10 * (z - 0.5)) ** -2
    ohm = 1.0 + (p.eta_contrast - 1.0) * z
    jsq = s.get("jsq", torch.zeros_like(r))
    X, Y = (lambda f: _d(f, 2, 1)), (lambda f: _d(f, 1, 1))
    ux, uy, vx, vy, wx, wy, tx, ty, rx, ry = X(u), Y(u), X(v), Y(v), X(w), Y(w), X(t), Y(t), X(r), Y(r)
    lap = lambda f: _d(f, 2, 2) + _d(f, 1, 2)  # noqa: E731
    wz, wzu, uzu, vzu = _z1(w, 1), _zup(w, 1, w), _zup(u, 2, w), _zup(v, 2, w)
    tz, tzu, tzz = _z1(t, 5), _zup(t, 5, w), _z2(t, 0)
    div = ux + vy + wz
    td = -r * (u * tx + v * ty + w * tzu) + p.gamma * ck * (kap * (lap(t) + tzz) + dkap * tzu) + p.f * p.zeta * ck * gm * ohm * jsq
    td = td - gm * t * div * r + sck * gm * (2 * (ux ** 2 + vy ** 2 + wz ** 2 - div ** 2 / 3)
                                             + (uy + vx) ** 2 + (wx + uzu) ** 2 + (wy + vzu) ** 2)
    m = [p.f / 2 * x * x for x in b]
    visc = sck / 3
    ud = -t * rx - r * tx - r * (u * ux + v * uy + w * uzu) + sck * (_z2(u, 3) + lap(u)) \
        + X(visc * div + m[0] - m[1] - m[2]) + Y(p.f * b[0] * b[1]) + _z1(p.f * b[0] * b[2], 5)
    vd = -t * ry - r * ty - r * (u * vx + v * vy + w * vzu) + sck * (_z2(v, 3) + lap(v)) \
        + Y(visc * div + m[1] - m[0] - m[2]) + X(p.f * b[0] * b[1]) + _z1(p.f * b[1] * b[2], 5)
    wd = -r * tz + p.theta * (p.cm + 1) * r - r * (u * wx + v * wy + w * wzu) + sck * lap(w) \
        + X(p.f * b[0] * b[2]) + Y(p.f * b[1] * b[2]) + _z1(visc * (ux + vy) + m[2] - m[0] - m[1], 2) + _z1(4 * visc * wz, 5)
    rz, rzu = _z1(r, 0), _zup(r, 0, w)
    for k in (0, p.nz - 1):      # no vertical acceleration at the walls
        rz[k] = rzu[k] = wd[k] / t[k]
    return [-u * rx - v * ry - r * div - w * rzu, td / r, ud / r, vd / r, (wd - t * rz) / r]


def _sd(h, dim, length=4.0):
    """Derivative of a halfcomplex spectrum along dim: f'_k = (i k) f_k."""
    n = h.shape[dim]
    i = torch.arange(n, device="cuda")
    k = torch.where(i <= n // 2, i, n - i).double() * (2 * math.pi / length)
    sgn = torch.where((i == 0) | (2 * i == n), 0.0, torch.where(2 * i < n, -1.0, 1.0)).double()
    return h.index_select(dim, (n - i) % n) * (k * sgn).reshape([-1 if d == dim else 1 for d in range(3)])


def _mag(p, s):
    """Induction in potentials, and B and |J|^2 of the potentials (no mean
    horizontal field, no mean vertical field stored)."""
    u, v, w, bx, by, bz, pol, tor = (s[n] for n in ("u", "v", "w", "bx", "by", "bz", "pol", "tor"))
    S = lambda f: _fwd(_fwd(f, 2), 1)     # noqa: E731
    I = lambda h: _inv(_inv(h, 2), 1)     # noqa: E731
    e = [S(v * bz - w * by), S(w * bx - u * bz), S(u * by - v * bx)]
    k2 = []
    for n in (p.ny, p.nx):
        i = torch.arange(n, device="cuda")
        k2.append((torch.where(i <= n // 2, i, n - i).double() * (2 * math.pi / 4.0)) ** 2)
    kk = -(k2[0][:, None] + k2[1][None, :])[None]
    inv = torch.where(kk == 0, torch.zeros_like(kk), 1.0 / kk)
    z = torch.linspace(0, 1, p.nz, dtype=torch.float64, device="cuda")[:, None, None]
    eta = p.zeta * p.ck * (1.0 + (p.eta_contrast - 1.0) * z)
    deta = p.zeta * p.ck * (p.eta_contrast - 1.0)
    w1 = _sd(e[0], 2) + _sd(e[1], 1)
    pd = eta * (pol * kk + _z2(pol, 3)) + (_sd(e[0], 1) - _sd(e[1], 2)) * inv
    td = eta * (tor * kk + _z2(tor, 3)) - _z1(w1, 5) * inv + e[2] + deta * _z1(tor, 5)
    dz = _z1(pol, 5)
    b = [I(_sd(dz, 2) + _sd(tor, 1)), I(_sd(dz, 1) - _sd(tor, 2)), I(-pol * kk)]
    jz = I(-tor * kk)
    j = jz ** 2 + (I(_sd(-pol * kk, 1)) - _z1(b[1], 5)) ** 2 + (_z1(b[0], 5) - I(_sd(-pol * kk, 2))) ** 2
    return [pd, td] + b + [j]


def exact(case, seed):
    k = case["kind"]
    if k in ("ops", "transforms", "lines"):
        shape = (case["nz"], case["ny"], case["nx"])
        gen = _gen(seed)
        f = _horiz(gen, shape) + 1e-2 * _noise(gen, shape)
        if k == "ops":
            return [_d(f, 2, 1), _d(f, 2, 2), _d(f, 1, 1), _d(f, 1, 2), _d(f, 2, 1), _d(f, 1, 1), _z1(f, 5), _z2(f, 3)]
        if k == "transforms":
            return [_fwd(_fwd(f, 2), 1), f, _dealias(_dealias(f, 2), 1)]
        f = f.float().double()
        return [o for dim in (2, 1) for o in (_d(f, dim, 1), _d(f, dim, 2), _dealias(f, dim))]
    if k == "rhs":
        p = _params(case)
        s = _fields(p, seed)
        s.update(_spectra(p, seed))
        return _hydro(p, s) + (_mag(p, s) if p.f else [])
    return None    # whole runs: their blocks are the cases above
