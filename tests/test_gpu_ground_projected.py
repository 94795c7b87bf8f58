"""The ground state's projected matrix: tridiagonal to rounding, and solved as such, on ordinary
bases; not tridiagonal where the Krylov space runs out or nearly so (couplings of 1, 1e-6 and
1e-11), and solved in full there.  Against numpy's eigenvalues of the same matrix."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


@pytest.mark.parametrize("phase", [1.0, 1j])
@pytest.mark.parametrize("weak", [1.0, 1e-6, 1e-11])
@pytest.mark.parametrize("n", [2, 3, 9, 40, 64, 126])
def test_chain(api, n, weak, phase):
    hop = [weak if i % 3 == 2 else 1.0 for i in range(n - 1)]
    H = api.Operator(n, [([i, i + 1 | api.CREATION], h * phase) for i, h in enumerate(hop)]
                     + [([i + 1, i | api.CREATION], h * np.conj(phase)) for i, h in enumerate(hop)]
                     + [([i, i | api.CREATION], 0.1 * ((7 * i) % 11)) for i in range(n)])
    b, _ = api.Basis.from_bytes(n, api.dets_to_bytes(["0" * i + "1" + "0" * (n - 1 - i) for i in range(n)], n))
    M = api.OperatorToDeterminantMatrix(H, b)
    w = np.linalg.eigvalsh(M)
    X, E = api.EigensystemOnBasis(H, b, 1, {"Zero": 1e-14})
    x = X.cpu().numpy()[:, 0]
    # a variance of 1e-14 leaves a residual of 1e-7 and an energy error below 1e-7
    assert abs(np.linalg.norm(x) - 1.0) < 1e-12
    assert np.linalg.norm(M @ x - E[0] * x) < 1.1e-7
    assert abs(E[0] - (x.conj() @ M @ x).real) < 1e-12
    assert -1e-12 < E[0] - w[0] < (1e-10 if weak == 1.0 else 1.1e-7)
