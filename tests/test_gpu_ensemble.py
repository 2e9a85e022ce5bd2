"""Batched 2D vorticity ensembles against the FP64 oracle (rhs2d,
rk4_step2d, initialize2d): every member of a mixed-size ensemble after a few
IF-RK4 steps, in all three execution modes (graph, plain, one member at a
time), which must agree bit for bit."""
import numpy as np
import pytest

import speccodelib_gb300 as S
from oracle import spectral_ref as R
from _util import rel_l2

pytestmark = pytest.mark.gpu

SIZES = [64, 128, 256, 128, 64]


def params(n):
    kmax = 2.0 * (n // 2) / 3.0
    dt = 0.5 / n
    return dt, 1.0 / (kmax ** 8 * dt)


NVAR = {S.SC_FP32: 6, S.SC_FP64: 2}


def oracle_steps(n, w, dt, nu, steps):
    p = R.Params2D(n=n, alpha=0.01, nu8=nu, dt=dt)
    for _ in range(steps):
        w = R.rk4_step2d(w, p)
    return w


@pytest.mark.parametrize("prec,tol", [(S.SC_FP64, 1e-12), (S.SC_FP32, 1e-5)])
def test_ensemble_matches_oracle(specns_lib, prec, tol):
    """Every compiled launch shape (pinned with set_variant), in all three
    modes; the modes agree bit for bit within a shape."""
    dts, nus = zip(*[params(n) for n in SIZES])
    seeds = [-(i + 1) for i in range(len(SIZES))]
    init = [R.initialize2d(n, s) for n, s in zip(SIZES, seeds)]
    ref = [oracle_steps(n, init[m], dts[m], nus[m], 3) for m, n in enumerate(SIZES)]
    for v in range(NVAR[prec]):
        outs = {}
        for mode in (0, 1, 2):
            with S.Ensemble2D(SIZES, dts, nus, 0.01, prec) as e:
                e.set_variant(v)
                e.init(seeds)
                for m, n in enumerate(SIZES):
                    assert rel_l2(e.get_member(m), init[m]) < (1e-14 if prec == S.SC_FP64 else 1e-6)
                e.rk4_steps(3, mode)
                outs[mode] = [e.get_member(m) for m in range(len(SIZES))]
                if mode == 0:
                    assert e.uses_graph()
                assert e.variant()[0] == v
        for m, n in enumerate(SIZES):
            assert rel_l2(outs[0][m], ref[m]) < tol, (v, m, n)
            assert np.array_equal(outs[0][m], outs[1][m]) and np.array_equal(outs[0][m], outs[2][m])


@pytest.mark.parametrize("prec,tol", [(S.SC_FP64, 1e-12), (S.SC_FP32, 1e-5)])
def test_ensemble_large_members(specns_lib, prec, tol):
    """N = 512 and 1024 members (the 16- and 32-point-per-lane x rows)."""
    sizes = [1024, 512]
    dts, nus = zip(*[params(n) for n in sizes])
    seeds = [-7, -8]
    for v in range(NVAR[prec]):
        with S.Ensemble2D(sizes, dts, nus, 0.01, prec) as e:
            e.set_variant(v)
            e.init(seeds)
            init = [e.get_member(m) for m in range(2)]
            e.rk4_steps(2)
            out = [e.get_member(m) for m in range(2)]
        for m, n in enumerate(sizes):
            w0 = init[m].astype(np.complex128)
            assert rel_l2(w0, R.initialize2d(n, seeds[m])) < (1e-14 if prec == S.SC_FP64 else 1e-6)
            assert rel_l2(out[m], oracle_steps(n, R.initialize2d(n, seeds[m]), dts[m], nus[m], 2)) < tol, (v, n)


def test_ensemble_autotuner(specns_lib):
    """The tuner times every shape, keeps the fastest, and leaves the member
    states as they were; stepping afterwards equals the pinned shape."""
    dts, nus = zip(*[params(n) for n in SIZES])
    seeds = [-(i + 1) for i in range(len(SIZES))]
    with S.Ensemble2D(SIZES, dts, nus, 0.01, S.SC_FP32) as e:
        e.init(seeds)
        before = [e.get_member(m) for m in range(len(SIZES))]
        chosen = e.tune(2)
        v, shape, ms = e.variant()
        assert v == chosen and len(ms) == NVAR[S.SC_FP32] and all(t > 0 for t in ms)
        assert ms[v] == min(ms)
        assert shape["threads"] in (256, 512) and shape["radix"] in (4, 8)
        for m in range(len(SIZES)):
            assert np.array_equal(e.get_member(m), before[m])
        e.rk4_steps(2)
        tuned = [e.get_member(m) for m in range(len(SIZES))]
    with S.Ensemble2D(SIZES, dts, nus, 0.01, S.SC_FP32) as e:
        e.set_variant(chosen)
        e.init(seeds)
        e.rk4_steps(2)
        for m in range(len(SIZES)):
            assert np.array_equal(e.get_member(m), tuned[m])


def test_ensemble_energy_decays_without_forcing(specns_lib):
    n = 128
    dt, nu = params(n)
    with S.Ensemble2D([n, n], [dt, dt], [nu, nu], 0.01, S.SC_FP64) as e:
        e.init([-3, -4])
        e0 = [R.energy2d(e.get_member(m)) for m in range(2)]
        e.rk4_steps(20)
        e1 = [R.energy2d(e.get_member(m)) for m in range(2)]
    assert all(abs(a - 0.5) < 1e-12 for a in e0)
    assert all(b < a for a, b in zip(e0, e1))


def test_many_members_of_one_size(specns_lib):
    """More members of one size than a grid's second dimension admits, in the
    launch-per-pass form: members at both ends equal to an ensemble of their own."""
    nm, n, var = 65540, 64, 5
    dt, nu = params(n)
    seeds = [-3, -5, -9]
    at = [0, 65535, nm - 1]
    with S.Ensemble2D([n] * 3, [dt] * 3, [nu] * 3, 0.01, S.SC_FP32) as e:
        e.set_variant(var)
        e.init(seeds)
        init = [e.get_member(m) for m in range(3)]
        e.rk4_steps(2)
        ref = [e.get_member(m) for m in range(3)]
    with S.Ensemble2D([n] * nm, [dt] * nm, [nu] * nm, 0.01, S.SC_FP32) as e:
        e.set_variant(var)
        for m, w in zip(at, init):
            e.set_member(m, w)
        e.rk4_steps(2, 1)
        for m, w in zip(at, ref):
            assert np.array_equal(e.get_member(m), w)
        assert not np.any(e.get_member(1)) and not np.any(e.get_member(nm - 2))


@pytest.mark.parametrize("prec,var,sizes", [(S.SC_FP32, 5, [64] * 128), (S.SC_FP32, 5, [1024] * 6),
                                            (S.SC_FP64, 1, [128] * 40), (S.SC_FP64, 1, [1024] * 4)])
def test_classes_of_many_tiles(specns_lib, prec, var, sizes):
    """Classes whose first pass takes each CTA through several tiles (its two
    buffers refilled, their barriers' phases turned): every member as when it
    runs alone, the first and the last as the oracle's."""
    n, nm = sizes[0], len(sizes)
    dt, nu = params(n)
    seeds = [-(m + 1) for m in range(nm)]
    outs = []
    for mode in (1, 2):
        with S.Ensemble2D(sizes, [dt] * nm, [nu] * nm, 0.01, prec) as e:
            e.set_variant(var)
            e.init(seeds)
            e.rk4_steps(1, mode)
            outs.append([e.get_member(m) for m in range(nm)])
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
    for m in (0, nm - 1):
        ref = oracle_steps(n, R.initialize2d(n, seeds[m]), dt, nu, 1)
        assert rel_l2(outs[0][m], ref) < (1e-12 if prec == S.SC_FP64 else 1e-5)


def test_member_read_into_fresh_and_odd_memory(specns_lib):
    """A member read into memory that was never touched, that starts and ends
    inside pages, and into pinned and device memory: the same values, and nothing
    beside them."""
    import ctypes as C
    import mmap
    torch = pytest.importorskip("torch")
    n = 512
    dt, nu = params(n)
    size = n * (n // 2 + 1) * 8
    with S.Ensemble2D([n], [dt], [nu], 0.01, S.SC_FP32) as e:
        e.init([-3])
        ref = e.get_member(0).tobytes()
        for shift in (0, 8, 4096 - 24):
            m = mmap.mmap(-1, size + 2 * 65536)
            p = C.addressof(C.c_char.from_buffer(m))
            assert specns_lib.sc_ens_get_member(e.h, 0, C.c_void_p(p + shift)) == 0
            assert m[shift:shift + size] == ref
            assert not any(m[:shift]) and not any(m[shift + size:])
        for b in (torch.zeros(size + 16, dtype=torch.uint8).pin_memory(), torch.zeros(size + 16, dtype=torch.uint8, device="cuda")):
            assert specns_lib.sc_ens_get_member(e.h, 0, C.c_void_p(b.data_ptr() + 8)) == 0
            got = b.cpu().numpy()
            assert got[8:8 + size].tobytes() == ref and not got[:8].any() and not got[8 + size:].any()
            assert specns_lib.sc_ens_set_member(e.h, 0, C.c_void_p(b.data_ptr() + 8)) == 0
            assert e.get_member(0).tobytes() == ref
