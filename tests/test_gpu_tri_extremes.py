"""The two ends of the spectrum of every chain's tridiagonal matrix (the pole range of a spectrum):
lengths around the four-row steps of a count, couplings of very different sizes, decoupled and
empty chains, chains that end early, against LAPACK's eigenvalues."""
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


def _ends(a, b):
    w = np.linalg.eigvalsh(np.diag(a) + np.diag(b, 1) + np.diag(b, -1))
    return w[0], w[-1]


@pytest.mark.parametrize("early", [0, 1])
@pytest.mark.parametrize("scale", [1e-150, 1.0, 1e120])
@pytest.mark.parametrize("ntri", [1, 2, 3, 4, 5, 8, 33, 200, 701])
def test_ends(api, ntri, scale, early):
    eng = api.engine()
    rng = np.random.default_rng(ntri)
    ns = 7
    A = rng.normal(size=(ns, ntri + 1)) * scale
    B = np.abs(rng.normal(size=(ns, ntri))) * scale
    A[1] += 300 * scale
    B[2] *= 10.0 ** rng.uniform(-20, 0, size=ntri)  # couplings from 1 down to 1e-20
    B[3, ntri // 2:] = 0.0                           # a chain that ends half way, zeros behind
    A[3, ntri // 2 + 1:] = 0.0
    B[4, 1:] = 0.0                                   # decoupled
    A[5], B[5] = 0.0, 0.0                            # nothing at all
    A[6], B[6] = 2.5 * scale, scale                  # the uniform chain
    got = np.zeros((ns, 2))
    eng.check(eng.L.qg_tri_extremes(eng.ctx, ns, ntri, api._ptr(A), api._ptr(B), early, api._ptr(got)))
    for s in range(ns):
        zero = np.flatnonzero(B[s, 1:] == 0.0)
        m = int(zero[0]) + 1 if early and len(zero) else ntri
        w = _ends(A[s, 1:m + 1], B[s, 1:m])
        norm = np.abs(A[s]).max() + 2 * np.abs(B[s]).max()
        # both sides are backward stable: a few eps of the norm, LAPACK's growing with the order
        assert np.abs(got[s] - w).max() <= (16 + ntri) * 2.2e-16 * norm


def test_bad_arguments(api):
    eng = api.engine()
    x = np.zeros(4)
    assert eng.L.qg_tri_extremes(eng.ctx, 1, 0, api._ptr(x), api._ptr(x), 0, api._ptr(x)) != 0
    assert eng.L.qg_tri_extremes(eng.ctx, 1, 1, C.c_void_p(), api._ptr(x), 0, api._ptr(x)) != 0
    assert eng.L.qg_tri_extremes(eng.ctx, 0, 1, C.c_void_p(), C.c_void_p(), 0, C.c_void_p()) == 0
