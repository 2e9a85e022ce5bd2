"""GPU parity of single kernels at the sizes where their tiling, remainders and
dispatch rules can go wrong, against the FP64 oracle."""
import numpy as np
import pytest

import speccodelib_gb300 as S
from oracle import spectral_ref as R
from _util import fresh, hermitian_fields, rel_l2

pytestmark = pytest.mark.gpu

DT = {S.SC_FP64: np.complex128, S.SC_FP32: np.complex64}


# Per-point products carry a few roundings of the field's precision (2^-24,
# 2^-53); the transform behind max |u| is held to 1e-5 / 1e-12 as elsewhere.
@pytest.mark.parametrize("prec,tol,tol_u", [(S.SC_FP64, 1e-13, 1e-12), (S.SC_FP32, 1e-6, 1e-5)])
@pytest.mark.parametrize("shape", [(8, 8, 8), (64, 16, 8), (128, 8, 32), (256, 32, 8), (512, 8, 16), (1024, 8, 8),
                                   (16, 64, 256)])
def test_diagnostics_shapes(specns_lib, shape, prec, tol, tol_u):
    """Every kx remainder, single rows (k = 0, n/2) and row pairs of both
    strided axes, and the lengths with and without a fused c2r maximum."""
    nx, ny, nz = shape
    v = [fresh(a, DT[prec]) for a in hermitian_fields(shape, 29)]
    vd = [a.astype(np.complex128) for a in v]
    kx, ky, kz, k2 = R.wavenumber(nx, ny, nz)
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz)) as h:
        h.set_state(*v)
        d, eks = h.diagnostics()
    assert abs(d["energy"] / R.energy(vd) - 1) < tol
    assert abs(d["enstrophy"] / R.enstrophy(vd, k2) - 1) < tol
    assert abs(d["max_div"] / R.max_divergence(vd, kx, ky, kz) - 1) < 10 * tol
    assert abs(d["max_u"] / R.max_velocity(vd, nx) - 1) < tol_u
    ref = R.spectrum(vd, k2, nx)
    assert np.abs(eks - ref).max() <= tol * ref.max()
    assert d["nonfinite"] == 0


@pytest.mark.parametrize("shape", [(32, 16, 8), (128, 16, 8)])
def test_diagnostics_nonfinite(specns_lib, shape):
    nx, ny, nz = shape
    v = [fresh(a, np.complex64) for a in hermitian_fields(shape, 5)]
    v[1][nz - 1, ny - 2, 3] = np.nan
    v[2][0, 0, nx // 2] = np.inf
    with S.SpectralNS(S.default_params(nx, S.SC_FP32, ny=ny, nz=nz)) as h:
        h.set_state(*v)
        with pytest.raises(S.SpecNSError) as e:
            h.diagnostics()
    assert e.value.code == 3


TOL = {S.SC_FP64: 1e-12, S.SC_FP32: 1e-5}   # the library's bounds against the oracle
X_SHAPES = [(16, 8, 8), (32, 8, 16), (64, 16, 8), (128, 8, 8), (256, 8, 16), (512, 8, 8), (1024, 8, 8)]


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("shape", X_SHAPES)
@pytest.mark.parametrize("sgs", ["none", "smag"])
def test_rhs_x_lengths(specns_lib, shape, prec, sgs):
    """The x-pass of the right-hand side (Lamb product; Lamb product and
    Smagorinsky stress) at every row length, on grids of few rows."""
    nx, ny, nz = shape
    kw = dict(forced=0) if sgs == "none" else dict(forced=0, sgs=S.SC_SGS_SMAG, c1=0.03)
    v = [fresh(a, DT[prec]) for a in hermitian_fields(shape, 41, kcut=0.4 * max(shape))]
    g = R.Grid(R.Params(nx=nx, ny=ny, nz=nz, forced=False, sgs=sgs, c1=0.03))
    ref = R.ratesdudt([a.astype(np.complex128) for a in v], g)
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz, **kw)) as h:
        h.set_state(*v)
        w = h.rhs()
    assert rel_l2(w, ref) < TOL[prec]


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("shape", X_SHAPES[1:6])
def test_vjp_x_lengths(specns_lib, shape, prec):
    """The adjoint's x-pass at the same lengths, over one RK4 step."""
    nx, ny, nz = shape
    v = [fresh(a, DT[prec]) for a in hermitian_fields(shape, 43, kcut=6.0)]
    lam = [fresh(a, DT[prec]) for a in hermitian_fields(shape, 44)]
    g = R.Grid(R.Params(nx=nx, ny=ny, nz=nz, nu=0.02, dt=1e-3))
    ref = R.rk4_step_adj([a.astype(np.complex128) for a in v], [a.astype(np.complex128) for a in lam], g)
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz, nu=0.02, dt=1e-3)) as h:
        h.set_state(*v)
        out = h.adjoint_vjp(1, lam, 1)
    assert rel_l2(out, ref) < (1e-11 if prec == S.SC_FP64 else 1e-4)   # the bounds of the adjoint's other tests


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("shape", [(16, 8, 8), (32, 64, 16), (64, 16, 256), (128, 8, 512), (32, 32, 1024)])
def test_kx0_copy(specns_lib, shape, prec):
    """symmetrize's kx = 0 copies between the pencils ky and -ky, with the
    forcing band on them, from a field without that symmetry: the right-hand
    side and two RK4 steps (fused stages and the last one)."""
    nx, ny, nz = shape
    v = [fresh(0.05 * a, DT[prec]) for a in hermitian_fields(shape, 51, kcut=5.0)]
    skew = [0.3 * a[:, :, 0] for a in hermitian_fields(shape, 52, kcut=4.0)]
    for a, s in zip(v, skew):
        a[:, :, 0] += (1j * s).astype(a.dtype)
    kw = dict(nu=0.02, dt=1e-3, fkmax=3.1, eps=0.2)
    g = R.Grid(R.Params(nx=nx, ny=ny, nz=nz, **kw))
    vd = [a.astype(np.complex128) for a in v]
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz, **kw)) as h:
        h.set_state(*v)
        w = h.rhs()
        h.rk4_steps(2)
        out = h.get_state()
    ref = R.ratesdudt(vd, g)
    assert rel_l2(w, ref) < TOL[prec]
    assert rel_l2([a[:, :, 0] for a in w], [a[:, :, 0] for a in ref]) < TOL[prec]
    ref = R.rk4_run(vd, g, 2)
    assert rel_l2(out, ref) < TOL[prec]
    assert rel_l2([a[:, :, 0] for a in out], [a[:, :, 0] for a in ref]) < TOL[prec]


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("shape,fk", [((32, 8, 8), 2.5), ((32, 128, 16), 40.0), ((128, 16, 32), 20.0), ((64, 16, 64), 2.5),
                                      ((16, 128, 128), 64.5)])
def test_short_z_pencils(specns_lib, shape, fk, prec):
    """The z kernels of short pencils (groups of threads, one component each):
    forced RK4 steps and their adjoint, with bands of fewer and more rows than a
    warp and of more than one kx tile."""
    nx, ny, nz = shape
    v = [fresh(0.05 * a, DT[prec]) for a in hermitian_fields(shape, 53, kcut=6.0)]
    lam = [fresh(a, DT[prec]) for a in hermitian_fields(shape, 54)]
    vd, ld = ([a.astype(np.complex128) for a in x] for x in (v, lam))
    kw = dict(nu=0.02, dt=1e-3, fkmax=fk, eps=0.2)
    g = R.Grid(R.Params(nx=nx, ny=ny, nz=nz, **kw))
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz, **kw)) as h:
        h.set_state(*v)
        out = h.adjoint_vjp(1, lam, 1)
        h.set_state(*v)
        h.rk4_steps(2)
        got = h.get_state()
    assert rel_l2(got, R.rk4_run(vd, g, 2)) < (1e-11 if prec == S.SC_FP64 else 1e-5)   # as the steps' other tests
    assert rel_l2(out, R.rk4_step_adj(vd, ld, g)) < (1e-11 if prec == S.SC_FP64 else 1e-4)


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("shape", [(16, 8, 256), (32, 8, 512), (16, 8, 1024)])
def test_vjp_long_z_pencils(specns_lib, shape, prec):
    """The adjoint's z-forward on long pencils: resident tiles (groups of threads)
    to 512 points, two tiles in flight beyond; band of more than one kx tile."""
    nx, ny, nz = shape
    v = [fresh(0.05 * a, DT[prec]) for a in hermitian_fields(shape, 55, kcut=6.0)]
    lam = [fresh(a, DT[prec]) for a in hermitian_fields(shape, 56)]
    kw = dict(nu=0.02, dt=1e-3, fkmax=9.0, eps=0.2)
    g = R.Grid(R.Params(nx=nx, ny=ny, nz=nz, **kw))
    ref = R.rk4_step_adj([a.astype(np.complex128) for a in v], [a.astype(np.complex128) for a in lam], g)
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz, **kw)) as h:
        h.set_state(*v)
        out = h.adjoint_vjp(1, lam, 1)
    assert rel_l2(out, ref) < (1e-11 if prec == S.SC_FP64 else 1e-4)   # the bounds of the adjoint's other tests


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("shape", [(8, 8, 8), (32, 16, 64), (512, 8, 32)])
@pytest.mark.parametrize("shift", [0, 4])
def test_device_state_round_trip(specns_lib, shape, prec, shift):
    """States in device memory, on the element's alignment and off it."""
    torch = pytest.importorskip("torch")
    nx, ny, nz = shape
    n = nz * ny * (nx // 2 + 1)
    cs = 8 if prec == S.SC_FP32 else 16
    bufs = [torch.zeros(n * cs + 16, dtype=torch.uint8, device="cuda") for _ in range(6)]
    rng = np.random.default_rng(3)
    v = [(rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(DT[prec]) for _ in range(3)]
    for b, a in zip(bufs, v):
        b[shift:shift + n * cs] = torch.from_numpy(a.view(np.uint8)).cuda()
    torch.cuda.synchronize()
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz)) as h:
        h.set_state_device(*(b.data_ptr() + shift for b in bufs[:3]))
        host = h.get_state()
        h.get_state_device(*(b.data_ptr() + shift for b in bufs[3:]))
    for a, b, c in zip(v, host, bufs[3:]):
        assert np.array_equal(b.reshape(-1), a)
        assert np.array_equal(c[shift:shift + n * cs].cpu().numpy().view(DT[prec]), a)
        assert int(c[:shift].sum()) == 0 and int(c[shift + n * cs:].sum()) == 0


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("shape", [(8, 16, 8), (16, 8, 32), (32, 8, 16), (64, 16, 8), (128, 8, 64), (256, 8, 8),
                                   (512, 8, 16), (1024, 8, 8), (32, 32, 512)])
def test_scalar_passes_shapes(specns_lib, shape, prec):
    """The scalar's flux in the velocity's passes at every row length (warp,
    lane-group and block x-pass), both forced scalar solvers; and with the
    kx = 0 copy off its symmetric values."""
    nx, ny, nz = shape
    f = [fresh(0.05 * a, DT[prec]) for a in hermitian_fields(shape, 61, ncomp=4, kcut=4.0)]
    f[3][:, :, 0] *= DT[prec](1 + 0.2j)
    kw = dict(nu=0.02, dt=1e-3, eps=0.2)
    g = R.Grid(R.Params(nx=nx, ny=ny, nz=nz, **kw))
    fd = [a.astype(np.complex128) for a in f]
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz, **kw)) as h:
        h.set_state(*f[:3])
        h.set_scalar(f[3])
        h.rot_scalar_steps(3, om=2.0, fk1=1.0, fk2=2.5, pr=0.7, scalarforced=True, epsphi=0.05)
        rot = list(h.get_state()) + [h.get_scalar()]
        h.set_state(*f[:3])
        h.set_scalar(f[3])
        for dt in (1e-3, 8e-4, 1.2e-3):
            h.ab2v_scalar_pass(dt, 0.7, True, 0.4)
        var = list(h.get_state()) + [h.get_scalar()]
    v, phi, _, _ = R.rot_scalar_run(fd[:3], fd[3], g, 3, 2.0, 1.0, 2.5, 0.7, True, 0.05)
    assert rel_l2(rot[:3], v) < TOL[prec]
    assert rel_l2(rot[3], phi) < TOL[prec]
    v, phi, _, _ = R.ab2v_scalar_run(fd[:3], fd[3], g, (1e-3, 8e-4, 1.2e-3), 0.7, True, 0.4)
    assert rel_l2(var[:3], v) < TOL[prec]
    assert rel_l2(var[3], phi) < TOL[prec]


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("shape", [(32, 256, 8), (32, 8, 256), (64, 512, 16), (128, 16, 512), (32, 1024, 8),
                                   (64, 8, 1024), (256, 64, 32), (512, 8, 64)])
def test_les_passes(specns_lib, shape, prec):
    """The y and z passes of the LES right-hand side at every tile shape, with
    a forcing band several tiles wide, one RK4 step, and a right-hand side
    without symmetrize (a variable-step pass)."""
    nx, ny, nz = shape
    kw = dict(nu=0.01, dt=1e-3, fkmax=6.2, eps=0.3, c1=0.03)
    v = [fresh(0.05 * a, DT[prec]) for a in hermitian_fields(shape, 71, kcut=8.0)]
    vd = [a.astype(np.complex128) for a in v]
    g = R.Grid(R.Params(nx=nx, ny=ny, nz=nz, sgs="smag", **kw))
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz, sgs=S.SC_SGS_SMAG, **kw)) as h:
        h.set_state(*v)
        w = h.rhs()
        h.rk4_steps(1)
        out = h.get_state()
        h.set_state(*v)
        h.ab2v_pass(1e-3)
        var = h.get_state()
    assert rel_l2(w, R.ratesdudt(vd, g)) < TOL[prec]
    assert rel_l2(out, R.rk4_run(vd, g, 1)) < TOL[prec]
    assert rel_l2(var, R.ab2v_run(vd, g, (1e-3,))[0]) < TOL[prec]


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("fk2", [1e5, 12.0])
def test_wide_rotating_band(specns_lib, fk2, prec):
    """Forcing bands as wide as the grid and wider, the squared upper bound past
    2^31 among them: the rotating solvers with and without a scalar."""
    nx, ny, nz = shape = (32, 16, 64)
    f = [fresh(0.05 * a, DT[prec]) for a in hermitian_fields(shape, 67, ncomp=4, kcut=6.0)]
    kw = dict(nu=0.02, dt=1e-3, eps=0.2)
    g = R.Grid(R.Params(nx=nx, ny=ny, nz=nz, **kw))
    fd = [a.astype(np.complex128) for a in f]
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz, **kw)) as h:
        h.set_state(*f[:3])
        h.set_scalar(f[3])
        h.rot_scalar_steps(2, om=2.0, fk1=1.0, fk2=fk2, pr=0.7, scalarforced=True, epsphi=0.05)
        both = list(h.get_state()) + [h.get_scalar()]
        h.set_state(*f[:3])
        h.rot_steps(2, om=2.0, fk1=1.0, fk2=fk2)
        alone = h.get_state()
    v, phi, _, _ = R.rot_scalar_run(fd[:3], fd[3], g, 2, 2.0, 1.0, fk2, 0.7, True, 0.05)
    assert rel_l2(both[:3], v) < TOL[prec]
    assert rel_l2(both[3], phi) < TOL[prec]
    assert rel_l2(alone, R.rot_run(fd[:3], g, 2, 2.0, 1.0, fk2)[0]) < TOL[prec]


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("shape", [(16, 8, 512), (256, 8, 512), (1024, 8, 512), (16, 16, 1024)])
def test_les_forcing_tiles(specns_lib, shape, prec):
    """The forcing coefficient of an LES right-hand side where the z-inverse sums
    the band in tiles of another width than the register kernel's, band wider
    than either: with and without the gradient form's row lengths."""
    nx, ny, nz = shape
    kw = dict(nu=0.01, dt=1e-3, fkmax=6.2, eps=0.3, c1=0.03)
    v = [fresh(0.05 * a, DT[prec]) for a in hermitian_fields(shape, 73, kcut=8.0)]
    ref = R.ratesdudt([a.astype(np.complex128) for a in v], R.Grid(R.Params(nx=nx, ny=ny, nz=nz, sgs="smag", **kw)))
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz, sgs=S.SC_SGS_SMAG, **kw)) as h:
        h.set_state(*v)
        w = h.rhs()
    assert rel_l2(w, ref) < TOL[prec]


@pytest.mark.parametrize("prec", [S.SC_FP64, S.SC_FP32])
@pytest.mark.parametrize("sgs", ["none", "smag"])
@pytest.mark.parametrize("shape", [(64, 16, 32), (64, 32, 64), (128, 16, 32), (128, 32, 64), (256, 16, 32), (256, 32, 64),
                                   (256, 64, 128), (512, 16, 32), (512, 32, 64)])
def test_x_row_counts(specns_lib, shape, sgs, prec):
    """The x-pass on either side of the row counts at which FP64 rows change
    from the block kernel to lane groups, and the LES from S_ij to gradients."""
    nx, ny, nz = shape
    kw = dict(nu=0.01, dt=1e-3, fkmax=3.1, eps=0.3)
    les = {} if sgs == "none" else dict(sgs=S.SC_SGS_SMAG, c1=0.03)
    v = [fresh(0.05 * a, DT[prec]) for a in hermitian_fields(shape, 79, kcut=8.0)]
    g = R.Grid(R.Params(nx=nx, ny=ny, nz=nz, sgs=sgs, c1=0.03, **kw))
    ref = R.ratesdudt([a.astype(np.complex128) for a in v], g)
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz, **kw, **les)) as h:
        h.set_state(*v)
        w = h.rhs()
    assert rel_l2(w, ref) < TOL[prec]


@pytest.mark.parametrize("shape", [(64, 16, 32), (64, 32, 64), (128, 32, 64), (256, 16, 32), (256, 32, 64), (512, 16, 32),
                                   (512, 32, 64)])
def test_vjp_row_counts(specns_lib, shape):
    """The adjoint's x-pass in FP64 on either side of its row count."""
    nx, ny, nz = shape
    v = [fresh(0.05 * a, np.complex128) for a in hermitian_fields(shape, 83, kcut=6.0)]
    lam = [fresh(a, np.complex128) for a in hermitian_fields(shape, 84)]
    kw = dict(nu=0.02, dt=1e-3)
    ref = R.rk4_step_adj(v, lam, R.Grid(R.Params(nx=nx, ny=ny, nz=nz, **kw)))
    with S.SpectralNS(S.default_params(nx, S.SC_FP64, ny=ny, nz=nz, **kw)) as h:
        h.set_state(*v)
        out = h.adjoint_vjp(1, lam, 1)
    assert rel_l2(out, ref) < 1e-11   # the bound of the adjoint's other tests


@pytest.mark.parametrize("where", ["device", "pinned"])
@pytest.mark.parametrize("lap", [0, 1])
def test_overlapping_state_buffers(specns_lib, where, lap):
    """A state read into buffers that overlap holds what copies in turn leave:
    one buffer for all three components (lap 0), or neighbours half over each
    other, from the last to the first in memory (lap 1)."""
    torch = pytest.importorskip("torch")
    nx, ny, nz = 128, 64, 64
    n = nz * ny * (nx // 2 + 1)
    rng = np.random.default_rng(4)
    v = [(rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64) for _ in range(3)]
    at = [0, 0, 0] if lap == 0 else [n, n // 2, 0]
    buf = torch.zeros(2 * n, dtype=torch.complex64, device="cuda") if where == "device" else \
        torch.zeros(2 * n, dtype=torch.complex64).pin_memory()
    torch.cuda.synchronize()
    with S.SpectralNS(S.default_params(nx, S.SC_FP32, ny=ny, nz=nz)) as h:
        h.set_state(*[a.reshape(nz, ny, nx // 2 + 1) for a in v])
        for _ in range(5):
            h.get_state_device(*(buf.data_ptr() + 8 * o for o in at))
            ref = np.zeros(2 * n, np.complex64)
            for o, a in zip(at, v):
                ref[o:o + n] = a
            assert np.array_equal(buf.cpu().numpy(), ref)


@pytest.mark.parametrize("prec,amp", [(S.SC_FP32, 1e18), (S.SC_FP64, 1e153)])
@pytest.mark.parametrize("nx", [16, 32, 64, 128, 256, 512, 1024])
def test_diagnostics_nonfinite_in_space(specns_lib, nx, prec, amp):
    """A field whose modes all have finite squares but whose velocity, all modes
    in phase at the origin, has not: only the count behind max |u| sees it."""
    ny = nz = 16
    v = [np.zeros((nz, ny, nx // 2 + 1), DT[prec]) for _ in range(3)]
    with S.SpectralNS(S.default_params(nx, prec, ny=ny, nz=nz)) as h:
        v[0][:4, :4, 1:5] = amp / 64           # 64 modes, |u| = 2 amp
        h.set_state(*v)
        assert h.diagnostics()[0]["nonfinite"] == 0
        v[0][:4, :4, 1:5] = amp                # |u| = 128 amp, its square beyond the type
        h.set_state(*v)
        with pytest.raises(S.SpecNSError) as e:
            h.diagnostics()
    assert e.value.code == 3


def test_calls_after_a_failed_allocation(specns_lib):
    """An error that one call has reported is not reported again by the next."""
    torch = pytest.importorskip("torch")
    n = 32
    v = [torch.zeros((n, n, n // 2 + 1), dtype=torch.complex64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    nm = 20000   # a terabyte of members
    with S.SpectralNS(S.default_params(n, S.SC_FP32)) as h:
        for use in (lambda: h.set_state_device(*(a.data_ptr() for a in v)), lambda: h.rk4_steps(1), h.get_state):
            with pytest.raises(S.SpecNSError) as e:
                S.Ensemble2D([1024] * nm, [1e-4] * nm, [0.0] * nm, 0.0, S.SC_FP64)
            assert e.value.code == 5
            use()
