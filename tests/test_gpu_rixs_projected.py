"""The Krylov-projected intermediate resolvent of the resonant spectra at every length of its
recursion (one vector, two, an incomplete space, the whole space and vectors past its end), against
dense linear algebra in numpy on all 120 determinants of 14 electrons in 16 spin-orbitals."""
import itertools

import numpy as np
import pytest

from conftest import golden

pytestmark = pytest.mark.gpu
# rounding of 1e-16 |H| (some 1e2) per step, through two resolvents of 2 / Gamma each: below 1e-11
TOL = 1e-8


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


@pytest.mark.parametrize("silent", [False, True])
@pytest.mark.parametrize("ntri", [1, 2, 5, 8, 24, 41, 60])
def test_projected_resolvent(api, ntri, silent):
    g = golden("rixs.json")
    op = lambda k: api.Operator.from_fixture(g[k])  # noqa: E731
    psi = api.Wavefunction.from_fixture(g["psi"][0])
    if silent:  # an absorption that gives nothing: the recursion is empty
        psi = api.Wavefunction(psi.nf, psi.det, psi.val * 0)
    dets = ["".join("0" if i in h else "1" for i in range(16)) for h in itertools.combinations(range(16), 2)]
    bas, _ = api.Basis.from_bytes(16, api.dets_to_bytes(dets, 16))
    M = {k: api.OperatorToDeterminantMatrix(op(k), bas) for k in ("H", "HX", "Tx", "Txd")}
    index = {bytes(b): i for i, b in enumerate(bas.dets_bytes())}
    v = np.zeros(len(dets), dtype=complex)
    for d, x in zip(psi.det, psi.val):
        v[index[bytes(d)]] = x
    o = {"Emin1": -5, "Emax1": 15, "NE1": 4, "Gamma1": 0.8, "Emin2": -2, "Emax2": 8, "NE2": 32, "Gamma2": 0.3,
         "E0_1": -3.0, "E0_2": -3.5, "DenseBorder": 0, "Epsilon": 1e-14, "NTri1": ntri, "NTri2": 80}
    G, st = api.CreateResonantSpectra(op("HX"), op("H"), op("Tx"), [op("Txd")], psi, o)
    assert st["method"] == "krylov" and np.isfinite(G).all()
    # an orthonormal basis of span{x, HX x, ...} of at most ntri vectors
    x = M["Tx"] @ v
    Q, w = [], x
    for _ in range(ntri):
        for _ in range(2):
            for q in Q:
                w = w - q * np.vdot(q, w)
        if np.linalg.norm(w) < 1e-8:
            break
        Q.append(w / np.linalg.norm(w))
        w = M["HX"] @ Q[-1]
    want = np.zeros((5, 33), dtype=complex)
    if Q:
        Q = np.array(Q).T
        for p in range(5):
            z = -5 + 20 * p / 4 - 3.0 + 0.4j
            mid = Q @ np.linalg.solve(z * np.eye(Q.shape[1]) - Q.conj().T @ M["HX"] @ Q, Q.conj().T @ x)
            y = M["Txd"] @ mid
            for i in range(33):
                z2 = -2 + 10 * i / 32 - 3.5 + 0.15j
                want[p, i] = np.vdot(y, np.linalg.solve(z2 * np.eye(120) - M["H"], y))
    assert G.shape == want.shape
    assert np.abs(G - want).max() <= TOL * max(np.abs(want).max(), 1e-300)
