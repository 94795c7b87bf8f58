"""Eigenvectors of groups of equal and nearly equal eigenvalues that are larger than the one-block
Gram-Schmidt takes (16): panels of 32 columns between and after the inverse iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("spread", [0.0, 1e-15, 1e-13, 1e-12, 1e-11, 1e-10])
@pytest.mark.parametrize("m", [17, 40, 64])
def test_large_groups(api, m, spread, cplx):
    """Two groups of m eigenvalues, each within m * spread, beside separated and clustered ones, in a
    dense rotated matrix."""
    rng = np.random.default_rng(m)
    k = 2 * m + 60
    B = rng.normal(size=(k, k)) + (1j * rng.normal(size=(k, k)) if cplx else 0.0)
    Q, _ = np.linalg.qr(B)
    d = np.concatenate([1.0 + spread * np.arange(m), 1.002 + spread * rng.random(m) * m,
                        1.003 + 3e-4 * np.arange(30), 2.0 + 0.5 * np.arange(30)])
    A = (Q * d) @ Q.conj().T
    A = (A + A.conj().T) / 2
    w, v = api.hermitian_eigh(A, k)
    scale = np.abs(d).max()
    # the bounds of the other eigensolver tests: eps times the order, with a margin
    assert np.abs(w - np.sort(d)).max() < 1e-13 * scale
    assert np.abs(A @ v - v * w).max() < 1e-12 * scale
    assert np.abs(v.conj().T @ v - np.eye(k)).max() < 1e-13
