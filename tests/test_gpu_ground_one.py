"""The ground state alone (one wanted state, every step on the device): real and complex
Hamiltonians, bases smaller than the first Krylov space and not a multiple of a row chunk,
against numpy's eigenvalues of the same matrix."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


def _impurity(api, nshell, holes, particles, cplx):
    from quanty_gb300 import workloads
    H, R, det, _ = workloads.anderson_impurity(nshell=nshell, hole_max=holes, particle_max=particles, field=0.1,
                                               complex_field=cplx)
    return H, api.closure(H, api.dets_to_bytes([det], H.nf), H.nf, R)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("nshell,holes,particles", [(0, 0, 0), (2, 1, 0), (2, 2, 0), (1, 0, 1)])
def test_ground_state(api, nshell, holes, particles, cplx):
    H, b = _impurity(api, nshell, holes, particles, cplx)
    w = np.linalg.eigvalsh(api.OperatorToDeterminantMatrix(H, b))
    X, E = api.EigensystemOnBasis(H, b, 1, {"Zero": 1e-14})
    x = X.cpu().numpy()[:, 0]
    # a variance of 1e-14 eV^2 leaves an error below variance / gap; energies are a few hundred eV
    assert abs(E[0] - w[0]) < 1e-10
    assert abs(np.linalg.norm(x) - 1.0) < 1e-12
    M = api.OperatorToDeterminantMatrix(H, b)
    assert np.linalg.norm(M @ x - E[0] * x) < 1.1e-7
    if not cplx:
        assert not np.any(x.imag)


def test_invariant_start(api):
    """A start vector that spans an invariant space alone: a diagonal operator, one determinant."""
    H = api.Operator(16, [([i, i | api.CREATION], float(i + 1)) for i in range(16)])
    b, _ = api.Basis.from_bytes(16, api.dets_to_bytes(["1" * 8 + "0" * 8], 16))
    X, E = api.EigensystemOnBasis(H, b, 1, {"Zero": 1e-14})
    assert abs(E[0] - 36.0) < 1e-13 and abs(abs(X.cpu().numpy()[0, 0]) - 1.0) < 1e-14
