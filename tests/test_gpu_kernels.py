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
