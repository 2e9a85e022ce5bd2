"""Performance cases: what a user of the library has it do, through its public
entry points (the handle API with the field resident in device memory, the 2D
ensembles, and the reference-signature operators on host arrays).

A case names a `kind` and its sizes.  The kinds:

  dns          n IF-RK4 steps of the forced DNS from a given field
  les          the same with the Smagorinsky or dynamic Smagorinsky stress
  rot_scalar   n passes of the rotating solver carrying a passive scalar
  ab2v_scalar  n passes of the variable-step AB2 carrying a passive scalar
  rot, ab2v    the same two solvers without the scalar
  adjoint      final-time shell enstrophy and its gradient over n RK4 steps
  ensemble     n steps of a batch of independent 2D vorticity runs
  diagnostics  FP64 energy, dissipation, CFL maximum and spectrum of a field
  operator     one reference subroutine on host arrays

Grids are powers of two per axis, as the library takes them; the ragged ones
have three different axis lengths.
"""
import ctypes

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import speccodelib_gb300 as S
from speccodelib_gb300 import specns as SP

EPS, FKMAX = 0.1, 2.5            # forcing: power 0.1 into k < 2.5
C1 = 0.17 ** 2                   # Smagorinsky constant squared
OM, FK1, FK2, PR, EPSPHI = 5.0, 1.0, 2.5, 0.7, 0.05
ALPHA = 0.01                     # linear damping of the 2D runs
SHELLS = (8, 16)                 # shells of the adjoint's enstrophy
AB2V_STEPS = (1.0, 0.8, 1.2, 0.9, 1.1)   # uneven steps, times the case's dt


def _grid(kind, name, nx, ny, nz, prec, steps, **more):
    return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, prec=prec, steps=steps, **more)


def listed():
    return [
        # a small field: a user's parameter scan or test run, where launches and latency count
        _grid("dns", "dns_64_f32", 64, 64, 64, "f32", 10),
        # the plain forced DNS at 128^3 in double precision, as the reference is built by default
        _grid("dns", "dns_128_f64", 128, 128, 128, "f64", 4),
        # an ordinary single-precision production grid
        _grid("dns", "dns_256_f32", 256, 256, 256, "f32", 4),
        # the largest: the 512^3 forced DNS
        _grid("dns", "dns_512_f32", 512, 512, 512, "f32", 2),
        # a ragged box: a long, a short and a middle axis
        _grid("dns", "dns_512x64x256_f32", 512, 64, 256, "f32", 5),
        # LES with the static model, 256^3
        _grid("les", "les_smag_256_f32", 256, 256, 256, "f32", 2, sgs="smag"),
        # LES with the dynamic model: ten steps hold one refresh of the coefficient
        _grid("les", "les_dyn_128_f32", 128, 128, 128, "f32", 10, sgs="dynsmag"),
        # rotating turbulence with a passive scalar, both forced
        _grid("rot_scalar", "rot_scalar_256_f32", 256, 256, 256, "f32", 4),
        # a passive scalar with a mean gradient and uneven steps, double precision
        _grid("ab2v_scalar", "ab2v_scalar_128_f64", 128, 128, 128, "f64", 4),
        # gradient of a final-time functional with respect to the initial field (forward and backward)
        _grid("adjoint", "adjoint_128_f32", 128, 128, 128, "f32", 20, every=10),
        # the batched 2D ensemble: 64 members of mixed size, advanced and read out
        dict(name="ensemble_64_f32", kind="ensemble", members="24x256 24x512 16x1024", prec="f32", steps=60),
        # what a solver evaluates every few steps: energy, dissipation, CFL maximum, E(k)
        _grid("diagnostics", "diagnostics_256_f32", 256, 256, 256, "f32", 1),
    ]


def draw(rng):
    """One more case: kinds, axis lengths, precision and step counts over the ranges above."""
    kind = rng.choice(["dns", "dns", "dns", "les", "rot_scalar", "ab2v_scalar", "rot", "ab2v", "adjoint", "ensemble",
                       "diagnostics", "operator"])
    prec = "f64" if rng.random() < 0.3 else "f32"
    if kind == "ensemble":
        sizes = sorted(rng.sample([64, 128, 256, 512, 1024], rng.randint(1, 3)))
        return dict(kind=kind, members=" ".join("%dx%d" % (rng.randint(1, 19), n) for n in sizes), prec="f32",
                    steps=rng.randint(1, 60))
    steps = rng.randint(1, 9)
    # cells times steps: a double-precision or multi-field step costs more
    cost = {"dns": 1, "les": 2, "rot_scalar": 1, "ab2v_scalar": 1, "rot": 1, "ab2v": 1, "adjoint": 4,
            "diagnostics": 1, "operator": 8}[kind] * (16 if prec == "f64" else 1)
    while True:
        nx, ny, nz = (1 << rng.randint(5, 9) for _ in range(3))
        if 1 << 15 <= nx * ny * nz and nx * ny * nz * steps * cost <= 1 << 27:
            break
    case = dict(kind=kind, nx=nx, ny=ny, nz=nz, prec=prec, steps=steps)
    if kind == "les":
        case["sgs"] = rng.choice(["smag", "dynsmag"])
    if kind == "adjoint":
        case["every"] = rng.randint(1, steps)
    if kind == "operator":
        case["op"] = rng.choice(["convecphi", "projection", "smag"])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dtype(case):
    return torch.complex64 if case["prec"] == "f32" else torch.complex128


def _prec(case):
    return S.SC_FP32 if case["prec"] == "f32" else S.SC_FP64


def _flow(case):
    """nu, dt of a case: the library's defaults on small grids, finer on large ones."""
    if case["kind"] == "les":
        return 1e-4, 1e-3
    return (1.5e-3, 5e-4) if max(case["nx"], case["ny"], case["nz"]) >= 256 else (0.01, 2e-3)


def _wave(nx, ny, nz, dev):
    """kx, ky, kz shaped to broadcast over (nz, ny, nx/2+1), and k^2, in double."""
    f = dict(dtype=torch.float64, device=dev)
    kx = torch.arange(nx // 2 + 1, **f)[None, None, :]
    ky = torch.fft.fftfreq(ny, 1.0 / ny, **f)[None, :, None]
    kz = torch.fft.fftfreq(nz, 1.0 / nz, **f)[:, None, None]
    return kx, ky, kz, kx * kx + ky * ky + kz * kz


def _kcut(nx):
    return 2.0 * (nx // 2) / 3.0


def _noise(case, seed, count, dev):
    """`count` random-phase fields with the conjugate symmetry of a real field, in double."""
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = torch.randn((count, nz, ny, nx // 2 + 1, 2), generator=g, device=dev, dtype=torch.float32)
    return [_symmetrize(torch.view_as_complex(x.double())) for x in r]


def _fields(case, seed, dev, scalar=False):
    """A random-phase velocity of energy 0.5 (k^4 exp(-2 (k/4)^2), or k^(-5/3) for the LES) truncated
    at 2/3, solenoidal unless it is there to be projected, and a scalar of the same shape; in the
    case's precision."""
    kx, ky, kz, k2 = _wave(case["nx"], case["ny"], case["nz"], dev)
    if case["kind"] == "les":
        amp = torch.where((k2 >= 4.0) & (k2 <= (case["nx"] / 3.0) ** 2), k2.clamp(min=1.0) ** (-11.0 / 12.0), 0.0 * k2)
    else:
        amp = torch.sqrt(k2) * torch.exp(-k2 / 16.0)
    amp = torch.where(k2 < _kcut(case["nx"]) ** 2, amp, 0.0 * amp)
    c = _noise(case, seed, 4 if scalar else 3, dev)
    v = c[:3] if case.get("op") == "projection" else _project(c[:3], kx, ky, kz, k2)
    v = [a * amp for a in v]
    q = sum(a.real ** 2 + a.imag ** 2 for a in v)
    e = q[..., 1:].sum() + 0.5 * q[..., 0].sum()
    out = [(a * torch.sqrt(0.5 / e)).to(_dtype(case)).contiguous() for a in v]
    if scalar:
        p = c[3] * amp
        q = p.real ** 2 + p.imag ** 2
        out.append((p * torch.sqrt(0.5 / (q[..., 1:].sum() + 0.5 * q[..., 0].sum()))).to(_dtype(case)).contiguous())
    return out


def _members(case):
    """Sizes of an ensemble's members, from "24x256 24x512 16x1024"."""
    out = []
    for part in case["members"].split():
        n, size = part.split("x")
        out += [int(size)] * int(n)
    return out


def _dt2(n):
    return 0.5 / n               # CFL about 0.5 at |u| ~ 1


def _nu8(n):
    return 1.0 / (_kcut(n) ** 8 * _dt2(n))


def _vorticities(case, seed, dev):
    """Random vorticity with E(k) ~ k exp(-(k/6)^2) and energy 0.5, one (N, N/2+1) field per member."""
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    out = []
    for n in _members(case):
        kx, ky, k2 = _wave2(n, dev)
        r = torch.randn((n, n // 2 + 1, 2), generator=g, device=dev, dtype=torch.float32)
        w = _symmetrize2(torch.view_as_complex(r.double()))
        k2s = k2.clamp(min=1.0)
        w = w * torch.where(k2 < _kcut(n) ** 2, torch.sqrt(k2s) * torch.exp(-0.5 * k2 / 36.0), 0.0 * k2)
        q = (w.real ** 2 + w.imag ** 2) / k2s
        out.append((w * torch.sqrt(0.5 / (q[:, 1:].sum() + 0.5 * q[:, 0].sum()))).to(_dtype(case)))
    return out


def _wave2(n, dev):
    f = dict(dtype=torch.float64, device=dev)
    kx = torch.arange(n // 2 + 1, **f)[None, :]
    ky = torch.fft.fftfreq(n, 1.0 / n, **f)[:, None]
    return kx, ky, kx * kx + ky * ky


def _params(case):
    nu, dt = _flow(case)
    sgs = {None: S.SC_SGS_NONE, "smag": S.SC_SGS_SMAG, "dynsmag": S.SC_SGS_DYNSMAG}[case.get("sgs")]
    return S.default_params(case["nx"], _prec(case), ny=case["ny"], nz=case["nz"], nu=nu, dt=dt, eps=EPS, fkmax=FKMAX,
                            sgs=sgs, c1=C1)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def prepare(case, seed):
    dev = torch.device("cuda")
    kind = case["kind"]
    st = dict(case=case)
    if kind == "ensemble":
        sizes = _members(case)
        st["ens"] = S.Ensemble2D(sizes, [_dt2(n) for n in sizes], [_nu8(n) for n in sizes], ALPHA, _prec(case))
        for m, w in enumerate(_vorticities(case, seed, dev)):
            st["ens"].set_member(m, w.cpu().numpy())
        return st
    scalar = kind in ("rot_scalar", "ab2v_scalar") or (kind == "operator" and case["op"] == "convecphi")
    f = _fields(case, seed, dev, scalar)
    if kind == "operator":
        st["host"] = [a.cpu().numpy() for a in f]
        st["out"] = np.empty_like(st["host"][0])
        return st
    st["in"] = f
    st["out"] = [torch.empty_like(a) for a in f]
    st["h"] = S.SpectralNS(_params(case))
    torch.cuda.synchronize()
    if kind in ("adjoint", "diagnostics"):       # these leave the handle's state as it is
        st["h"].set_state_device(*(a.data_ptr() for a in f))
    return st


def _scalar_call(name, h, t):
    SP._check(getattr(SP.lib(), name)(h.h, ctypes.c_void_p(t.data_ptr())))


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "ensemble":
        st["ens"].rk4_steps(case["steps"])
        return [st["ens"].get_member(m) for m in range(len(st["ens"].n))]
    if kind == "operator":
        nx, f = case["nx"], st["host"]
        if case["op"] == "convecphi":
            S.convecphi_dns(f[0], f[1], f[2], f[3], st["out"], nx)
            return st["out"]
        if case["op"] == "projection":           # in place, and the identity on its own result
            S.projection(*f)
            return f
        return S.smag(f[0], f[1], f[2], delta=np.pi / _kcut(nx), c1=C1)
    h = st["h"]
    if kind == "diagnostics":
        d, eks = h.diagnostics()
        return dict(d, spectrum=eks)
    if kind == "adjoint":
        J, grad = h.adjoint(case["steps"], case["every"], *SHELLS)
        return dict(J=J, grad=list(grad))
    h.set_state_device(*(a.data_ptr() for a in st["in"][:3]))
    scalar = kind in ("rot_scalar", "ab2v_scalar")
    if scalar:
        _scalar_call("sc_set_scalar", h, st["in"][3])
    if kind in ("dns", "les"):
        h.rk4_steps(case["steps"])
    elif kind == "rot":
        h.rot_steps(case["steps"], OM, FK1, FK2)
    elif kind == "rot_scalar":
        h.rot_scalar_steps(case["steps"], OM, FK1, FK2, PR, True, EPSPHI)
    else:
        dt = _flow(case)[1]
        for i in range(case["steps"]):
            if scalar:
                h.ab2v_scalar_pass(dt * AB2V_STEPS[i % 5], PR, True, 1.0)
            else:
                h.ab2v_pass(dt * AB2V_STEPS[i % 5])
    h.get_state_device(*(a.data_ptr() for a in st["out"][:3]))
    if scalar:
        _scalar_call("sc_get_scalar", h, st["out"][3])
    return st["out"]


def work(case):
    """Each input read and each output written once; 2.5 N log2 N flops per real transform."""
    cb = 8 if case["prec"] == "f32" else 16
    kind = case["kind"]
    if kind == "ensemble":
        sizes = _members(case)
        pts = sum((n // 2 + 1) * n for n in sizes)
        return {"bytes": 2.0 * cb * pts,
                "flops": case["steps"] * 4.0 * 5 * sum(2.5 * n * n * np.log2(n * n) for n in sizes)}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    fb = float(cb * (nx // 2 + 1) * ny * nz)
    tr = 2.5 * nx * ny * nz * np.log2(float(nx * ny * nz))
    if kind == "operator":
        io, n = {"convecphi": (5, 7), "projection": (6, 0), "smag": (9, 12)}[case["op"]]
        return {"bytes": io * fb, "flops": n * tr}
    if kind == "diagnostics":
        return {"bytes": 3 * fb, "flops": 3 * tr}
    if kind == "adjoint":
        return {"bytes": 6 * fb, "flops": case["steps"] * 4 * (9 + 15) * tr}
    fields = 8 if kind in ("rot_scalar", "ab2v_scalar") else 6
    n = {"dns": 4 * 9, "les": 4 * 21, "rot": 9, "ab2v": 9, "rot_scalar": 13, "ab2v_scalar": 13}[kind] * case["steps"]
    if case.get("sgs") == "dynsmag":
        n += 42 * ((case["steps"] + 9) // 10)
    return {"bytes": fields * fb, "flops": n * tr}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _c2r(c, nx):
    return torch.fft.irfft(torch.fft.ifft2(c, dim=(0, 1), norm="forward"), n=nx, dim=2, norm="forward")


def _r2c(r):
    """Transform of a physical field, times 1/N."""
    return torch.fft.fft2(torch.fft.rfft(r, dim=2, norm="forward"), dim=(0, 1), norm="forward")


def _symmetrize(c):
    """Zero the Nyquist planes and the mean; make the kx = 0 plane conjugate-symmetric."""
    nz, ny, nxh = c.shape
    keep = torch.ones((nz, ny, 1), dtype=torch.float64, device=c.device)
    keep[:, ny // 2] = 0.0
    keep[nz // 2] = 0.0
    first = keep[..., 0].clone()
    first[0, 0] = 0.0
    p = c[..., 0] * first
    src = torch.conj(torch.roll(torch.flip(p, (0, 1)), (1, 1), (0, 1)))
    tgt = torch.zeros((nz, ny), dtype=torch.bool, device=c.device)
    tgt[nz // 2 + 1:] = True
    tgt[0, ny // 2 + 1:] = True
    p = torch.where(tgt, src, p)
    return torch.cat([p[..., None], c[..., 1:nxh - 1] * keep, torch.zeros_like(c[..., :1])], dim=2)


def _symmetrize2(w):
    n, nxh = w.shape
    w = w.clone()
    w[n // 2] = 0.0
    w[:, nxh - 1] = 0.0
    w[0, 0] = 0.0
    w[n // 2 + 1:, 0] = torch.conj(torch.flip(w[1:n // 2, 0], (0,)))
    return w


def _project(w, kx, ky, kz, k2):
    t = (kx * w[0] + ky * w[1] + kz * w[2]) / k2.clamp(min=1.0)
    return [w[0] - kx * t, w[1] - ky * t, w[2] - kz * t]


def _lamb(v, nx, kx, ky, kz):
    w = [1j * (ky * v[2] - kz * v[1]), 1j * (kz * v[0] - kx * v[2]), 1j * (kx * v[1] - ky * v[0])]
    u = [_c2r(a, nx) for a in v]
    w = [_c2r(a, nx) for a in w]
    return [_r2c(u[(c + 1) % 3] * w[(c + 2) % 3] - u[(c + 2) % 3] * w[(c + 1) % 3]) for c in range(3)]


def _energy(v, band):
    q = sum(a.real ** 2 + a.imag ** 2 for a in v) * band
    return q[..., 1:].sum() + 0.5 * q[..., 0].sum()


def _strain(v, kx, ky, kz):
    return [1j * kx * v[0], 0.5j * (kx * v[1] + ky * v[0]), 0.5j * (kx * v[2] + kz * v[0]), 1j * ky * v[1],
            0.5j * (ky * v[2] + kz * v[1]), 1j * kz * v[2]]


def _norm(s):
    return torch.sqrt(2.0 * (s[0] ** 2 + s[3] ** 2 + s[5] ** 2 + 2.0 * (s[1] ** 2 + s[2] ** 2 + s[4] ** 2)))


def _pair(i):
    return ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))[i]


def _dynamic_cs2(v, nx, kx, ky, kz, k2, delta, ratio):
    """Germano-Lilly coefficient with box-averaged least squares, sharp test filter k <= kcut / ratio."""
    g = (k2 <= (_kcut(nx) / ratio) ** 2).double()
    s = [_c2r(a, nx) for a in _strain(v, kx, ky, kz)]
    sa = _norm(s)
    gs = [_c2r(g * a, nx) for a in _strain(v, kx, ky, kz)]
    ga = _norm(gs)
    u = [_c2r(a, nx) for a in v]
    gu = [_c2r(g * a, nx) for a in v]
    lm = mm = 0.0
    for i in range(6):
        a, b = _pair(i)
        L = _c2r(g * _r2c(u[a] * u[b]), nx) - gu[a] * gu[b]
        M = _c2r(g * _r2c(2.0 * delta ** 2 * sa * s[i]), nx) - 2.0 * (ratio * delta) ** 2 * ga * gs[i]
        wt = 1.0 if a == b else 2.0
        lm = lm + wt * (L * M).sum()
        mm = mm + wt * (M * M).sum()
    return lm / mm


def _rhs(v, case, wave, c1=None):
    kx, ky, kz, k2 = wave
    w = _lamb(v, case["nx"], kx, ky, kz)
    band = (k2 < FKMAX ** 2).double()
    a = EPS / (2.0 * _energy(v, band))
    w = [x + a * band * y for x, y in zip(w, v)]
    if c1 is not None:
        delta = np.pi / _kcut(case["nx"])
        s = [_c2r(x, case["nx"]) for x in _strain(v, kx, ky, kz)]
        sa = _norm(s)
        k = (kx, ky, kz)
        for i in range(6):
            p, q = _pair(i)
            t = _r2c(-2.0 * c1 * delta ** 2 * sa * s[i])
            w[p] = w[p] - 1j * k[q] * t
            if p != q:
                w[q] = w[q] - 1j * k[p] * t
    return _project([_symmetrize(x) for x in w], kx, ky, kz, k2)


def _rk4(v, case, wave, c1=None):
    nu, dt = _flow(case)
    k2 = wave[3]
    E = torch.exp(-nu * k2 * dt / 2)
    k1 = _rhs(v, case, wave, c1)
    kb = _rhs([E * (a + 0.5 * dt * b) for a, b in zip(v, k1)], case, wave, c1)
    kc = _rhs([E * a + 0.5 * dt * b for a, b in zip(v, kb)], case, wave, c1)
    kd = _rhs([E * E * a + E * dt * b for a, b in zip(v, kc)], case, wave, c1)
    keep = (k2 < _kcut(case["nx"]) ** 2).double()
    return [keep * (E * E * a + dt / 6.0 * (E * E * p + 2 * E * q + 2 * E * r + s))
            for a, p, q, r, s in zip(v, k1, kb, kc, kd)]


def _force_band(w, v, k2, lo2, hi2, power):
    band = ((k2 >= lo2) & (k2 < hi2)).double()
    a = power / (2.0 * _energy(v, band))
    return [x + a * band * y for x, y in zip(w, v)]


def _flux(v, phi, nx, kx, ky, kz):
    """i k . (u phi)."""
    p = _c2r(phi, nx)
    f = [_r2c(_c2r(a, nx) * p) for a in v]
    return 1j * (kx * f[0] + ky * f[1] + kz * f[2])


def _helical(kx, ky, kz, k2):
    """Unit vectors of positive helicity at every mode."""
    s, k = np.sqrt(0.5), torch.sqrt(k2.clamp(min=1e-30))
    d2 = (ky * ky + kz * kz).expand_as(k2)
    d = torch.sqrt(d2.clamp(min=1e-30))
    one = torch.ones_like(k2)
    on = (d2 > 0).double()
    hx = s * 1j * on * d2 / k / d
    hy = s * (-kz * on / d - 1j * on * kx * ky / k / d) + s * (1 - on) * (kx * one > 0)
    hz = s * (ky * on / d - 1j * on * kz * kx / k / d) + s * 1j * (1 - on) * (kx * one > 0)
    return hx, hy, hz


def _rotating(f, case, wave, scalar):
    """The helical-wave AB2: an Euler half step, a midpoint restart, then AB2."""
    kx, ky, kz, k2 = wave
    nx, ny = case["nx"], case["ny"]
    nu, dt = _flow(case)
    v, phi = f[:3], f[3] if scalar else None
    h = _helical(*wave)
    ph = 2.0 * dt * kz * OM / torch.sqrt(k2.clamp(min=1e-30)) * (k2 > 0)
    e = (torch.exp(torch.complex(-nu * k2 * dt, ph)), torch.exp(torch.complex(-nu * k2 * dt, -ph)))
    sq = [torch.sqrt(x) for x in e]
    basis = ([torch.conj(x) for x in h], h)
    ep = torch.exp(-nu * k2 * dt / PR)

    def dot(a, b):
        return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

    amp = [dot(v, b) for b in basis]
    start, phi0, old, ophi = list(amp), phi, None, None
    for i in range(case["steps"]):
        w = _lamb(v, nx, kx, ky, kz)
        w = _force_band(w, v, k2, *((FK1, FK2) if scalar else (FK1 ** 2, FK2 ** 2)), EPS)
        keep = (k2 < ny * ny / 9.0).double() if scalar else 1.0
        w = _project([keep * _symmetrize(x) for x in w], kx, ky, kz, k2)
        if scalar:
            wphi = _force_band([_flux(v, phi, nx, kx, ky, kz)], [phi], k2, FK1 ** 2, FK2 ** 2, EPSPHI)[0]
            wphi = keep * _symmetrize(wphi)
        if i == 0:
            amp = [(a + 0.5 * dt * dot(w, b)) * s for a, b, s in zip(amp, basis, sq)]
            phi = (phi + 0.5 * dt * wphi) * torch.sqrt(ep) if scalar else None
        elif i == 1:
            amp = [a * x + dt * dot(w, b) * s for a, b, s, x in zip(start, basis, sq, e)]
            phi = phi0 * ep + dt * wphi * torch.sqrt(ep) if scalar else None
        else:
            amp = [(a + 0.5 * dt * (3.0 * dot(w, b) - x * dot(old, b))) * x for a, b, x in zip(amp, basis, e)]
            phi = (phi + 0.5 * dt * (3.0 * wphi - ophi * ep)) * ep if scalar else None
        if i != 1:
            old = w
            ophi = wphi if scalar else None
        v = [amp[0] * a + amp[1] * torch.conj(a) for a in h]
        if not scalar:
            v = [(k2 < _kcut(nx) ** 2) * a for a in v]
    return v + ([phi] if scalar else [])


def _variable_ab2(f, case, wave, scalar):
    """The variable-step AB2; with the scalar no truncation, and phi as its own first history."""
    kx, ky, kz, k2 = wave
    nu, base = _flow(case)
    v, phi = f[:3], f[3] if scalar else None
    v0, phi0, old, ophi, dto = v, phi, None, None, 0.0
    for i in range(case["steps"]):
        dt = base * AB2V_STEPS[i % 5]
        if scalar:
            w = _rhs(v, case, wave)
            wphi = _symmetrize(_flux(v, phi, case["nx"], kx, ky, kz) - v[2])
        else:
            band = (k2 < FKMAX ** 2).double()
            w = _lamb(v, case["nx"], kx, ky, kz)
            a = EPS / (2.0 * _energy(v, band))
            w = _project([x + a * band * y for x, y in zip(w, v)], kx, ky, kz, k2)
        e1, e0 = torch.exp(-nu * k2 * dt), torch.exp(-nu * k2 * dto)
        p1, p0 = torch.exp(-nu * k2 * dt / PR), torch.exp(-nu * k2 * dto / PR)
        r = dt / dto if i else 0.0
        if i == 0:
            v = [(a + dt * b) * e1 for a, b in zip(v, w)]
            phi = (phi + dt * wphi) * p1 if scalar else None
            old, ophi, dto = w, phi, dt
        elif i == 1:
            s, ek, dl = 0.5 * (1 + r * r), 0.5 * (1 - r * r), 0.5 * dto * (1 + r) ** 2
            v = [(s * z * e0 + ek * a + dl * b) * e1 for z, a, b in zip(v0, v, w)]
            phi = (s * phi0 * p0 + ek * phi + dl * wphi) * p1 if scalar else None
            dto = dt + dto
        else:
            s, ek = (1 + 0.5 * r) * dt, -0.5 * r * dt
            v = [(a + s * b + ek * c * e0) * e1 for a, b, c in zip(v, w, old)]
            if scalar:
                phi, ophi = (phi + s * wphi + ek * ophi * p0) * p1, wphi
            old, dto = w, dt
        if not scalar:
            keep = ((k2 < _kcut(case["nx"]) ** 2) & (k2 > 0)).double()
            v = [keep * a for a in v]
    return v + ([phi] if scalar else [])


def _shell_enstrophy(v, k2):
    ll = torch.floor(torch.sqrt(k2) + 0.5)
    return _energy(v, k2 * ((ll >= SHELLS[0]) & (ll <= SHELLS[1])))


def _vorticity_step(w, n, dev):
    kx, ky, k2 = _wave2(n, dev)
    inv = torch.where(k2 > 0, 1.0 / k2.clamp(min=1.0), 0.0 * k2)
    keep = (k2 < _kcut(n) ** 2).double()
    dt = _dt2(n)
    E = torch.exp(-(ALPHA + _nu8(n) * k2 ** 4) * dt / 2)

    def real(c):
        return torch.fft.irfft(torch.fft.ifft(c, dim=0, norm="forward"), n=n, dim=1, norm="forward")

    def spec(r):
        return torch.fft.fft(torch.fft.rfft(r, dim=1, norm="forward"), dim=0, norm="forward")

    def rhs(s):
        u, v, o = real(1j * ky * inv * s), real(-1j * kx * inv * s), real(s)
        return keep * _symmetrize2(-1j * (kx * spec(u * o) + ky * spec(v * o)))

    k1 = rhs(w)
    kb = rhs(E * (w + 0.5 * dt * k1))
    kc = rhs(E * w + 0.5 * dt * kb)
    kd = rhs(E * E * w + E * dt * kc)
    return E * E * w + dt / 6.0 * (E * E * k1 + 2 * E * kb + 2 * E * kc + kd)


def exact(case, seed):
    dev = torch.device("cuda")
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        for n, w in zip(_members(case), _vorticities(case, seed, dev)):
            w = w.to(torch.complex128)
            for _ in range(case["steps"]):
                w = _vorticity_step(w, n, dev)
            out.append(w.cpu().numpy())
        return out
    nx = case["nx"]
    scalar = kind in ("rot_scalar", "ab2v_scalar") or (kind == "operator" and case["op"] == "convecphi")
    f = [a.to(torch.complex128) for a in _fields(case, seed, dev, scalar)]
    wave = _wave(nx, case["ny"], case["nz"], dev)
    kx, ky, kz, k2 = wave
    if kind == "dns":
        for _ in range(case["steps"]):
            f = _rk4(f, case, wave)
        return f
    if kind == "les":
        c1 = C1
        for i in range(case["steps"]):
            if case["sgs"] == "dynsmag" and i % 10 == 0:
                c1 = _dynamic_cs2(f, nx, kx, ky, kz, k2, np.pi / _kcut(nx), 2.0)
            f = _rk4(f, case, wave, c1)
        return f
    if kind in ("rot", "rot_scalar"):
        return _rotating(f, case, wave, scalar)
    if kind in ("ab2v", "ab2v_scalar"):
        return _variable_ab2(f, case, wave, scalar)
    if kind == "operator":
        if case["op"] == "convecphi":
            out = _flux(f[:3], f[3], nx, kx, ky, kz)
            return out.cpu().numpy()
        if case["op"] == "projection":
            out = _project(f, kx, ky, kz, k2)
        else:
            s = [_c2r(a, nx) for a in _strain(f, kx, ky, kz)]
            sa = _norm(s)
            out = [_r2c(-2.0 * C1 * (np.pi / _kcut(nx)) ** 2 * sa * a) for a in s]
        return [a.cpu().numpy() for a in out]
    if kind == "diagnostics":
        q = sum(a.real ** 2 + a.imag ** 2 for a in f)
        q[..., 0] *= 0.5
        ll = torch.floor(torch.sqrt(k2) + 0.5).long()
        eks = torch.zeros(nx // 2 + 2, dtype=torch.float64, device=dev)
        eks.scatter_add_(0, ll.clamp(max=nx // 2 + 1).reshape(-1), q.reshape(-1))
        u2 = sum(_c2r(a, nx) ** 2 for a in f)
        ens = float((k2 * q).sum())
        return dict(energy=float(q.sum()), enstrophy=ens, dissipation=2.0 * _flow(case)[0] * ens, max_div=None,
                    max_u=float(torch.sqrt(u2.max())), nonfinite=0.0, cs2=None, mm=None, lm=None,
                    spectrum=eks[1:nx // 2 + 1].cpu().numpy())
    # adjoint: dJ/dRe + i dJ/dIm of every stored coefficient, by reverse-mode differentiation
    v0 = [a.clone().requires_grad_(True) for a in f]
    v = v0
    for _ in range(case["steps"]):
        v = checkpoint(lambda *s: tuple(_rk4(list(s), case, wave)), *v, use_reentrant=False)
    J = _shell_enstrophy(v, k2)
    grad = torch.autograd.grad(J, v0)
    return dict(J=float(J.detach()), grad=[a.cpu().numpy() for a in grad])
