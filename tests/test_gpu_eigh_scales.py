"""The ends of the scale: tridiagonal chains whose norm is near or below the smallest normal number, and
the zero matrix, whose eigenvectors are any orthonormal set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


@pytest.mark.parametrize("exponent", [-970, -1000, -1020, -1030, -1050])
@pytest.mark.parametrize("ntri", [2, 5, 33])
def test_smallest_chains(api, ntri, exponent):
    eng = api.engine()
    rng = np.random.default_rng(ntri)
    a, b = rng.normal(size=(3, ntri + 1)), np.abs(rng.normal(size=(3, ntri)))
    A, B = np.ldexp(a, exponent), np.ldexp(b, exponent)  # below 2^-1022 rounded to multiples of 2^-1074
    got = np.zeros((3, 2))
    eng.check(eng.L.qg_tri_extremes(eng.ctx, 3, ntri, api._ptr(A), api._ptr(B), 0, api._ptr(got)))
    for s in range(3):
        up = np.ldexp(A[s, 1:], -exponent), np.ldexp(B[s, 1:], -exponent)
        w = np.linalg.eigvalsh(np.diag(up[0]) + np.diag(up[1], 1) + np.diag(up[1], -1))[[0, -1]]
        norm = np.abs(up[0]).max() + 2 * np.abs(up[1]).max()
        # a few eps of the norm on both sides, and the spacing of the numbers that the result is rounded to
        assert np.abs(np.ldexp(got[s], -exponent) - w).max() <= (16 + ntri) * 2.2e-16 * norm + np.ldexp(1.0, -1074 - exponent)


@pytest.mark.parametrize("k", [8, 41, 60, 200])
def test_zero_matrix(api, k):
    w, v = api.hermitian_eigh(np.zeros((k, k), dtype=complex), k)
    assert np.abs(w).max() <= 1e-290
    assert np.abs(v.conj().T @ v - np.eye(k)).max() < 1e-13
