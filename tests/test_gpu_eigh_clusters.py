"""Eigenvectors of dense spectra on the device: spectra whose neighbours all lie within 1e-3 of the
norm, so the whole set is one cluster and the block Gram-Schmidt runs, at the edges of its panels
(32 columns, 16 x 16 tiles) and of the one-block form (16), with tight groups and equal values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


def _check(api, A, d, nv):
    k = len(d)
    w, v = api.hermitian_eigh(A, nv)
    scale = max(1.0, np.abs(d).max())
    # the bounds of the other eigensolver tests: eps times the order, with a margin
    assert np.abs(w - np.sort(d)).max() < 1e-13 * scale
    assert np.abs(A @ v - v * w[:nv]).max() < 1e-12 * scale
    assert np.abs(v.conj().T @ v - np.eye(nv)).max() < 1e-13


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m", [15, 16, 17, 31, 32, 33, 48, 49, 65, 300])
def test_one_cluster(api, m, cplx):
    """m neighbours 1e-4 apart beside separated eigenvalues."""
    rng = np.random.default_rng(m)
    k = max(m + 12, 60)
    B = rng.normal(size=(k, k)) + (1j * rng.normal(size=(k, k)) if cplx else 0.0)
    Q, _ = np.linalg.qr(B)
    d = np.concatenate([np.arange(m) * 1e-4 * (1 + 0.1 * rng.random(m)), 1.0 + np.arange(k - m) * 0.5])
    A = Q @ np.diag(d) @ Q.conj().T
    A = (A + A.conj().T) / 2
    _check(api, A, d, k)
    _check(api, A, d, m)


@pytest.mark.parametrize("spread", [0.0, 1e-15, 1e-12, 1e-10, 1e-8])
def test_tight_groups_in_a_cluster(api, spread):
    """Forty groups of five inside one cluster, `spread` apart, and a matrix that is one multiple
    of the identity to rounding."""
    rng = np.random.default_rng(3)
    k = 200
    Q, _ = np.linalg.qr(rng.normal(size=(k, k)))
    d = np.repeat(np.arange(k // 5) * 3e-4, 5) + spread * rng.random(k)
    A = Q @ np.diag(d) @ Q.T + np.eye(k)
    A = (A + A.T) / 2
    _check(api, A, d + 1.0, k)
    _check(api, np.eye(k) * 2.0 + 0.0j, np.full(k, 2.0), k)
