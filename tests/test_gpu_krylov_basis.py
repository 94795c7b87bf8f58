"""The Krylov-basis Lanczos (full reorthogonalisation) on the device, real and complex, against the
recursion in numpy on the same matrix: coefficients, vectors, and the end of the list when the
space is exhausted."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


def _numpy(M, v, ntri, eps):
    n = len(v)
    K = np.zeros((ntri, n), dtype=complex)
    a, b = np.zeros(ntri + 1), np.zeros(ntri)
    err, w = 1.0, v.astype(complex)
    for i in range(ntri):
        if i:
            w = M @ K[i - 1]
            for j in range(i - 1, -1, -1):
                c = np.vdot(K[j], w)
                if j == i - 1:
                    a[i] = c.real
                w = w - c * K[j]
        b[i] = np.linalg.norm(w)
        x = w / b[i] if b[i] > 0 else 0 * w
        if i:
            if (np.abs(K[:i].conj() @ x) ** 2).sum() > eps:
                x = 0 * x
            err *= b[i] ** 2 / (b[i] ** 2 + 2.3e-308 + 2.220446049250313e-16 * a[i] ** 2)
        K[i] = np.where(np.abs(x) > eps / err, x, 0)
    a[ntri] = np.vdot(K[-1], M @ K[-1]).real
    return K, a, b


@pytest.mark.parametrize("vector", ["real", "imaginary", "complex"])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("nshell,holes,particles,ntri", [(0, 0, 0, 1), (0, 0, 0, 2), (1, 0, 1, 3), (2, 1, 0, 20), (1, 0, 1, 37)])
def test_krylov_lanczos(api, nshell, holes, particles, ntri, cplx, vector):
    from quanty_gb300 import workloads
    H, R, det, _ = workloads.anderson_impurity(nshell=nshell, hole_max=holes, particle_max=particles, field=0.1,
                                               complex_field=cplx)
    eng = api.engine()
    bas = api.closure(H, api.dets_to_bytes([det], H.nf), H.nf, R)
    n, eps = bas.n, 1e-10
    rng = np.random.default_rng(ntri)
    re, im = rng.normal(size=n), rng.normal(size=n)
    v = {"real": re + 0j, "imaginary": 1j * im, "complex": re + 1j * im}[vector]
    M = api.OperatorToDeterminantMatrix(H, bas)
    Kw, aw, bw = _numpy(M, v, ntri, eps)
    with eng.on_stream():
        x = eng.torch.from_numpy(v).cuda()
        K = eng.torch.zeros((ntri, n), dtype=eng.torch.complex128, device="cuda")
    a, b = np.zeros(ntri + 1), np.zeros(ntri)
    eng.check(eng.L.qg_lanczos_krylov(eng.ctx, H.handle(eng), bas.h, C.c_void_p(x.data_ptr()), ntri, eps,
                                      api._ptr(a), api._ptr(b), C.c_void_p(K.data_ptr())))
    Kd = eng.to_host(K)
    # full reorthogonalisation: rounding grows with the steps and the spread of H, not beyond
    assert np.abs(a - aw).max() < 1e-9 * np.abs(aw).max()
    assert np.abs(b - bw).max() < 1e-9 * np.abs(aw).max()
    assert np.abs(Kd - Kw).max() < 1e-8


def test_exhausted_space(api):
    """Eight determinants, twelve steps: the vectors past the space are empty, in the reference's
    single projection too."""
    H = api.Operator(8, [([i, (i + 1) % 8 | api.CREATION], 1.0) for i in range(8)]
                     + [([(i + 1) % 8, i | api.CREATION], 1.0) for i in range(8)]
                     + [([i, i | api.CREATION], 0.3 * i * i) for i in range(8)])
    eng = api.engine()
    dets = ["0" * i + "1" + "0" * (7 - i) for i in range(8)]
    bas, _ = api.Basis.from_bytes(8, api.dets_to_bytes(dets, 8))
    rng = np.random.default_rng(0)
    for v in (rng.normal(size=8) + 0j, rng.normal(size=8) + 1j * rng.normal(size=8)):
        with eng.on_stream():
            x = eng.torch.from_numpy(v).cuda()
            K = eng.torch.zeros((12, 8), dtype=eng.torch.complex128, device="cuda")
        a, b = np.zeros(13), np.zeros(12)
        eng.check(eng.L.qg_lanczos_krylov(eng.ctx, H.handle(eng), bas.h, C.c_void_p(x.data_ptr()), 12, 1e-10,
                                          api._ptr(a), api._ptr(b), C.c_void_p(K.data_ptr())))
        Kd = eng.to_host(K)
        assert all(np.any(Kd[i]) for i in range(8)) and not np.any(Kd[8:])
        assert np.abs(Kd[:8].conj() @ Kd[:8].T - np.eye(8)).max() < 1e-12
