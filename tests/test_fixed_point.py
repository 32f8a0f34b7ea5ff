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


def q_field(kind, nl, N):
    """noise or eddies, in all layers, in the top one alone (top), in the
    bottom one (bottom), weaker in each layer down (decay), or of single
    precision (single)."""
    rng, n = np.random.default_rng(nl), N - 1
    q = 1e-7 * rng.standard_normal((nl, n, n))
    if "eddies" in kind:
        x = 2 * np.pi * np.arange(n) / n
        for _ in range(8):
            a, b, c, d, e = rng.random(5)
            wave = np.outer(np.sin((1 + int(12 * a)) * x + 6 * b), np.sin((1 + int(12 * c)) * x + 6 * d))
            q += 2e-6 * e * wave * 0.6 ** np.arange(nl)[:, None, None]
    if "single" in kind:
        q = q.astype(np.float32).astype(float)
    if "decay" in kind:
        q *= 0.6 ** np.arange(nl)[:, None, None]
    if "top" in kind:
        q[1:] = 0
    if "bottom" in kind:
        q[:-1] = 0
    return q


def projection_errors(lib, modes, q, N):
    """Of psi (a row a layer: FP64 sums, fixed point), from the projections of
    an inversion alone, in units of 2^-53 of the layer's norm: layers to modes
    at the points, modes to layers at the rows' wave numbers."""
    l2m, m2l, ird = modes
    nl, k = len(ird), np.pi / 4e6 * np.arange(1, N)

    def project(mat, f):
        out = [np.empty((nl, N - 1, N - 1)) for _ in range(3)]
        mat, f = np.ascontiguousarray(mat), np.ascontiguousarray(f)
        lib.modes_errors.argtypes = [ctypes.c_int] * 3 + [ctypes.c_void_p] * 5
        lib.modes_errors(nl, N - 1, N - 1, mat.ctypes.data, f.ctypes.data, *(o.ctypes.data for o in out))
        return out

    def spectral(m):
        s = sf.dstn(m, type=1, axes=(1, 2)) / -(k[None, :, None] ** 2 + k[None, None] ** 2 + ird[:, None, None])
        return sf.idst(s, type=1, axis=1)
    *fwd, m = project(l2m, q)
    *back, psi = project(m2l, spectral(m))
    norm = np.linalg.norm(sf.idst(psi, type=1, axis=2), axis=(1, 2))
    return np.stack([np.linalg.norm(sf.idst(np.tensordot(m2l, spectral(f), 1) + b, type=1, axis=2), axis=(1, 2))
                     for f, b in zip(fwd, back)], 1) / norm[:, None] * 2.0 ** 53


@pytest.mark.parametrize("kind", ["noise", "noise top", "eddies top", "noise bottom", "noise single", "eddies single"])
@pytest.mark.parametrize("nl", [3, 8, 10])
def test_projection_error_no_larger_than_fp64(dstcore, qgwlib, nl, kind):  # noqa: F811
    """What the projections' rounding gives psi, also where products are
    exact (rest below the top layer, single precision), is no larger than
    with FP64 sums (or 2 units, the rounding of the results themselves)."""
    N = 128
    f64, fx = np.sqrt((projection_errors(dstcore, qgwlib.eigmode(C.cfg2(N, nl)), q_field(kind, nl, N), N) ** 2).mean(0))
    assert fx <= max(f64, 2.0), (f64, fx)


@pytest.mark.parametrize("kind", ["noise", "noise top", "noise decay", "noise bottom", "noise single", "eddies top",
                                  "eddies decay single"])
@pytest.mark.parametrize("nl,ratio", [(10, 1.3), (12, 1.5), (16, 1.3), (17, 1.3), (20, 1.3), (20, 1.5), (30, 1.3),
                                      (32, 1.3)])
def test_projection_error_of_every_layer(dstcore, qgwlib, nl, ratio, kind):  # noqa: F811
    """The same layer by layer, for graded profiles of many layers wherever
    the projections run in fixed point: their mean over the layers (each
    layer's within 2 units more, a draw of the roundings)."""
    dh = 4000 * (ratio - 1) / (ratio ** nl - 1) * ratio ** np.arange(nl)
    gp = 0.02 * 0.1 ** (np.arange(nl - 1) / (nl - 2))
    modes = qgwlib.eigmode(dict(C.cfg2(64, nl), dh=list(dh), N2=list(2 * gp / (dh[1:] + dh[:-1]))))
    if not all(dstcore.modes_fixed(nl, np.ascontiguousarray(m).ctypes.data_as(ctypes.c_void_p)) for m in modes[:2]):
        assert nl > 20 or ratio > 1.3
        return
    e = projection_errors(dstcore, modes, q_field(kind, nl, 64), 64)
    f64, fx = np.sqrt((e ** 2).mean(0))
    assert fx <= max(f64, 2.0) and np.all(e[:, 1] <= np.maximum(e[:, 0], 2.0) + 2.0), e


def vorticity(kind, N):
    rng, (Y, X) = np.random.default_rng(11), np.mgrid[1:N, 1:N]
    if kind == "front":
        return 1e-5 + 1e-6 * np.tanh((X - N / 2 + N / 16 * np.sin(12 * Y / N)) / 3)
    if kind == "vortex":
        return 1e-5 * np.exp(-((X - N / 3) ** 2 + (Y - N / 2) ** 2) / 50) + 1e-12 * rng.standard_normal(X.shape)
    q = sum(2e-6 * a * np.sin(2 * np.pi * int(1 + 4 * b) * X / N + 6 * c) * np.sin(2 * np.pi * int(1 + 4 * d) * Y / N + 6 * e)
            for a, b, c, d, e in rng.random((8, 5)))
    if kind == "single":
        return q.astype(np.float32).astype(float)
    return 1e-7 * rng.standard_normal(X.shape) + q * (kind == "eddies and noise") if "noise" in kind else q


@pytest.mark.parametrize("kind", ["noise", "eddies", "eddies and noise", "single", "front", "vortex"])
def test_jacobian_error_no_larger_than_fp64(dstcore, kind):  # noqa: F811
    N = 160
    q, k = vorticity(kind, N), np.pi / 4e6 * np.arange(1, N)
    psi = sf.idstn(sf.dstn(q, type=1) / -(k[:, None] ** 2 + k ** 2 + 1e-10), type=1)
    q, psi = (np.ascontiguousarray(np.pad(f, 1)) for f in (q, psi))
    e64, efx, exact = (np.empty((N - 1, N - 1)) for _ in range(3))
    dstcore.jacobian_errors.argtypes = [ctypes.c_int] * 2 + [ctypes.c_void_p] * 5
    dstcore.jacobian_errors(N - 1, N - 1, psi.ctypes.data, q.ctypes.data, *(e.ctypes.data for e in (e64, efx, exact)))
    f64, fx = (np.linalg.norm(e) / np.linalg.norm(exact) * 2.0 ** 53 for e in (e64, efx))
    assert fx <= max(f64, 2.0), (f64, fx)


@pytest.mark.gpu
@pytest.mark.parametrize("bc", [0.0, -1.0])
@pytest.mark.parametrize("kind", ["eddies", "single", "half"])
def test_jacobian_of_a_step(qgwlib, kind, bc):
    """A step of nothing but the Jacobian, so long that q itself is all but
    lost in it, against long double: to 4 units of 2^-53 (its own rounding, the
    coefficient's, the update's and the comparison's), and exactly zero where
    q is."""
    N = 96
    p = dict(C.cfg1(N), nl=1, dh=[4000.0], N2=[1.0], beta=0.0, tau0=0.0, nu=0.0, hEkb=0.0, bc_fac=bc, cfl=1e30)
    r = qgwlib.Run(p)
    q = np.zeros(r.shape)
    n = r.shape[2] - 2
    q[0, 1:-1, 1:-1] = vorticity("single" if kind == "single" else "eddies", n + 1)
    if kind == "half":
        q[0, :, : N // 2] = 0
    r.set_q(q)
    psi, q = r.get()
    dt = 1e18
    r.fix_dt(dt)
    r.step(1)
    q1 = r.get()[1][0, 1:-1, 1:-1]
    r.close()
    P, Q = (f[0].astype(np.longdouble) for f in (psi, q))

    def d(f, a, b):
        return (f[1 + a[1]:1 + a[1] + n, 1 + a[0]:1 + a[0] + n] - f[1 + b[1]:1 + b[1] + n, 1 + b[0]:1 + b[0] + n])
    o, E, W, S, T = (0, 0), (1, 0), (-1, 0), (0, -1), (0, 1)
    NE, NW, SE, SW = (1, 1), (-1, 1), (1, -1), (-1, -1)
    J = (d(Q, T, o) * (d(P, E, W) + d(P, NE, NW)) - d(Q, S, o) * (d(P, E, W) + d(P, SE, SW))
         - d(Q, E, o) * (d(P, T, S) + d(P, NE, SE)) + d(Q, W, o) * (d(P, T, S) + d(P, NW, SW))
         + d(Q, NE, o) * d(P, E, T) + d(Q, SE, o) * d(P, S, E) + d(Q, NW, o) * d(P, T, W) + d(Q, SW, o) * d(P, W, S))
    ref = Q[1:-1, 1:-1] - np.longdouble(dt) * 23 / 12 * J / (12 * np.longdouble(p["Lx"] / N) ** 2)
    assert np.linalg.norm((q1 - ref).astype(float)) <= 4 * 2.0 ** -53 * np.linalg.norm(ref.astype(float))
    if kind == "half":
        assert np.all(q1[:, 2: N // 2 - 2] == 0)


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
@pytest.mark.parametrize("nl", [8, 10, 16, 20, 24])
def test_inversion_of_one_layer(qgwlib, nl):
    """psi of a q in the top layer alone, whose other layers' products are
    exact, against scipy's transforms."""
    N = 256
    p = C.cfg2(N, nl)
    q = np.pad(q_field("noise top", nl, N), ((0, 0), (1, 1), (1, 1)))
    r = qgwlib.Run(p)
    r.set_q(q)
    psi, _ = r.get()
    r.close()
    l2m, m2l, ird = qgwlib.eigmode(p)
    k = np.pi * np.arange(1, N) / p["Lx"]
    s = sf.dstn(np.tensordot(l2m, q[:, 1:-1, 1:-1], 1), type=1, axes=(1, 2))
    s /= -(k[None, None] ** 2 + k[None, :, None] ** 2 + ird[:, None, None])
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
