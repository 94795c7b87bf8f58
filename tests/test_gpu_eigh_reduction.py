"""The tridiagonal reduction in one launch: orders around its grid (four rows per block up to one
block per SM, then more rows), real and complex, and complex orders too large for the blocks'
shared memory, which take a launch per column."""
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
@pytest.mark.parametrize("k", [41, 43, 44, 45, 255, 257, 591, 593, 609, 1100, 1201])
def test_reduction(api, k, cplx):
    rng = np.random.default_rng(k)
    B = rng.normal(size=(k, k)) + (1j * rng.normal(size=(k, k)) if cplx else 0.0)
    A = (B + B.conj().T) / 2
    nv = 3
    w, v = api.hermitian_eigh(A, nv)
    want = np.linalg.eigvalsh(A)
    scale = np.abs(want).max()
    # the bounds of the other eigensolver tests: eps times the order, with a margin
    assert np.abs(w - want).max() < 1e-13 * scale
    assert np.abs(A @ v - v * w[:nv]).max() < 1e-12 * scale
    assert np.abs(v.conj().T @ v - np.eye(nv)).max() < 1e-13
    if not cplx:
        assert not np.any(v.imag)


def test_reduced_columns(api):
    """Columns that are already in tridiagonal form (no reflector), and a block-diagonal matrix."""
    k = 64
    A = np.zeros((k, k))
    A[:40, :40] = np.diag(np.arange(40.0)) + np.diag(np.full(39, 0.5), 1) + np.diag(np.full(39, 0.5), -1)
    rng = np.random.default_rng(0)
    B = rng.normal(size=(24, 24))
    A[40:, 40:] = B + B.T
    w, v = api.hermitian_eigh(A + 0j, k)
    want = np.linalg.eigvalsh(A)
    assert np.abs(w - want).max() < 1e-13 * np.abs(want).max()
    assert np.abs(A @ v - v * w).max() < 1e-12 * np.abs(want).max()
    assert np.abs(v.conj().T @ v - np.eye(k)).max() < 1e-13
