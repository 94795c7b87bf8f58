"""Eigenvectors of many copies of one small block, each a little different: groups of 12 to 150
eigenvalues within 1e-14 to 1e-12 of the norm, whose inverse iterations come out close to dependent."""
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
@pytest.mark.parametrize("spread", [3e-14, 1e-13, 3e-13, 1e-12, 3e-12])
@pytest.mark.parametrize("m", [12, 20, 64, 150])
def test_copies_of_a_block(api, m, spread, cplx):
    for seed in range(3):
        rng = np.random.default_rng(1000 * m + seed)
        n0 = int(rng.integers(4, 7))
        B = rng.normal(size=(n0, n0)) + (1j * rng.normal(size=(n0, n0)) if cplx else 0.0)
        A = np.kron(np.eye(m), B + B.conj().T) + spread * np.diag(rng.random(n0 * m))
        w, v = api.hermitian_eigh(A, len(A))
        scale = np.abs(w).max()
        # the bounds of the other eigensolver tests; within a group vectors may mix over its width
        assert np.abs(v.conj().T @ v - np.eye(len(A))).max() < 1e-13
        assert np.abs(A @ v - v * w).max() < spread + 1e-13 * scale
