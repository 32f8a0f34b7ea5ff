"""The FP64 path's fixed-point DST-I (dst_fx.h): its work items on the host
against the definition, and whole inversions on the GPU at the lengths and
magnitudes where its rules change."""
import ctypes

import numpy as np
import pytest
import scipy.fft as sf

from qgw_gb300 import configs as C
from test_host import dstcore  # noqa: F401


def rows(M):
    rng, j = np.random.default_rng(M), np.arange(1, M)
    yield rng.standard_normal(M - 1)
    yield np.sin(np.pi * 3 * j / M) + 0.3 * np.sin(np.pi * 11 * j / M) + 1e-3 * rng.standard_normal(M - 1)
    yield np.exp(-((j - M / 3) / 4) ** 2) + 1e-9 * rng.standard_normal(M - 1)
    yield rng.standard_normal(M - 1) / j ** 2
    yield np.where((j == 1) | (j == M - 1), 1.0, 0.0) + 1e-12 * rng.standard_normal(M - 1)
    yield np.ones(M - 1)
    yield (-1.0) ** j
    yield rng.standard_normal(M - 1) * 1e-200
    yield rng.standard_normal(M - 1) * 1e200


@pytest.mark.parametrize("M", [4, 6, 10, 14, 16, 30, 70, 128, 240, 256, 384, 486, 512, 1000, 1024, 2048, 2430, 4096,
                               5, 9, 22, 33, 131, 207, 301, 514, 953, 1025, 2039])
def test_error_no_larger_than_fp64(dstcore, M):  # noqa: F811
    """Against the DST-I by its definition in long double, over random,
    smooth, peaked and decaying rows, the half-length forms and (from 5 on)
    the chirp-z ones: no row further off than the worst of
    the floating-point transform's rows (or 2 units of 2^-53, the rounding
    of the results and tables themselves), and all together closer."""
    dstcore.dst_fx_errors.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    err = np.zeros((0, 2))
    for x in rows(M):
        e, x = np.zeros(2), np.ascontiguousarray(x)
        dstcore.dst_fx_errors(M, x.ctypes.data, e.ctypes.data)
        err = np.vstack([err, e])
    f64, fx = err.T
    assert fx.max() <= max(f64.max(), 2.0), err
    assert np.sqrt((fx ** 2).mean()) <= max(np.sqrt((f64 ** 2).mean()), 1.0), err


def test_rows_of_zeros_and_non_finite_rows(dstcore):  # noqa: F811
    dstcore.dst_fx_run.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    x = np.zeros((4, 63))
    x[1, 5], x[2, 62], x[3, 7] = np.nan, np.inf, -0.0
    dstcore.dst_fx_run(64, 4, x.ctypes.data)
    assert np.all(x[[0, 3]] == 0) and np.all(np.isnan(x[[1, 2]]))


@pytest.mark.gpu
@pytest.mark.parametrize("NX,NY", [(4, 6), (10, 14), (128, 16), (16, 256), (256, 128), (512, 30), (30, 512),
                                   (1024, 12), (96, 1024), (2048, 64), (64, 2048), (2430, 8), (4096, 10)])
def test_inversion_at_transform_lengths(qgwlib, NX, NY):
    """psi of a random q against scipy's transforms, at the smallest sizes
    and at each compiled length along x and along y."""
    p = dict(C.cfg1(NX), NY=NY)
    q = C.noise_ic(p, 7)
    r = qgwlib.Run(p)
    r.set_q(q)
    psi, _ = r.get()
    r.close()
    l2m, m2l, ird = qgwlib.eigmode(p)
    m = np.tensordot(l2m, q[:, 1:-1, 1:-1], 1)
    k, l = np.pi * np.arange(1, NX) / p["Lx"], np.pi * np.arange(1, NY) / p["Lx"]
    s = sf.dstn(m, type=1, axes=(1, 2)) / -(k[None, None] ** 2 + l[None, :, None] ** 2 + ird[:, None, None])
    ref = np.tensordot(m2l, sf.idstn(s, type=1, axes=(1, 2)), 1)
    assert np.linalg.norm(psi[:, 1:-1, 1:-1] - ref) <= 2e-14 * np.linalg.norm(ref)


@pytest.mark.gpu
@pytest.mark.parametrize("e", [-700, 700])
def test_inversion_scales_with_q(qgwlib, e):
    """A power of two on q is one on psi, bit for bit."""
    p = dict(C.cfg2(96, 4), NY=128)
    q = C.noise_ic(p, 9)
    out = []
    for f in (1.0, 2.0 ** e):
        r = qgwlib.Run(p)
        r.set_q(q * f)
        out.append(r.get()[0] / f)
        r.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("bc", [0.0, 1.0, -1.0])
def test_rings(qgwlib, bc, prec):
    """The ring of fields taken out: wrapped, or at walls psi = 0 and
    q = 2 bc / Delta^2 psi at the adjacent point with corners of 0."""
    p = dict(C.cfg1(40), NY=40 if bc < 0 else 24, bc_fac=bc)
    r = qgwlib.Run(p, precision=prec)
    r.set_q(C.noise_ic(p, 5))
    psi, q = r.get()
    out = np.full(r.shape, np.nan)
    r.step_host(1, q, out)
    again = r.get()
    r.close()
    c = 2 * bc / (p["Lx"] / 40) ** 2
    for P, Q in ((psi, q), again, (again[0], out)):
        eP, eQ = (np.pad(F[:, 1:-1, 1:-1], ((0, 0), (1, 1), (1, 1)), "wrap" if bc < 0 else "constant") for F in (P, Q))
        if bc > 0:
            eQ[:, 0], eQ[:, -1], eQ[:, 1:-1, 0], eQ[:, 1:-1, -1] = (c * F for F in (
                P[:, 1], P[:, -2], P[:, 1:-1, 1], P[:, 1:-1, -2]))
        assert np.array_equal(P, eP)
        np.testing.assert_allclose(Q, eQ, rtol=1e-14, atol=0)
    assert np.array_equal(again[1], out)


@pytest.mark.gpu
@pytest.mark.parametrize("N,nl", [(1024, 6), (2048, 3)])
def test_transforms_in_place(qgwlib, N, nl):
    """1024 and 2048 points: the single run's transforms in one buffer, with
    blocks of one to six rows and a last block of fewer, against the
    ensemble's in two, bit for bit."""
    p = C.cfg2(N, nl)
    q = C.noise_ic(p, 13)
    ens = qgwlib.Ensemble([p], 0)
    ens.set_q(0, q)
    want = ens.get(0)[0]
    ens.step(2)
    want2 = ens.get(0)
    ens.close()
    for rows, cols in ((2, 4), (1, 2), (5, 4), (16, 4)):
        r = qgwlib.Run(p)
        r.set_shape(row_group_fwd=rows, row_group_inv=rows, col_tile=cols)
        r.set_q(q)
        assert np.array_equal(r.get()[0], want)
        r.step(2)
        psi, q2 = r.get()
        r.close()
        assert np.array_equal(psi, want2[0]) and np.array_equal(q2, want2[1]), rows
