"""One state where the Krylov space runs out: operators with one, two and a few distinct values on
more rows than the first Krylov space holds (101), and start vectors inside a block of their own.  The
state has to be normalised, an eigenvector, and the lowest of its space."""
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


def _basis(api, nf, electrons):
    from itertools import combinations
    dets = ["".join("1" if o in p else "0" for o in range(nf)) for p in combinations(range(nf), electrons)]
    return api.Basis.from_bytes(nf, api.dets_to_bytes(dets, nf))[0]


def _number(api, i, v):
    return [([i, i | api.CREATION], v)]


def _check(M, x, E, lowest):
    # a variance below 1e-14 is a residual below 1e-7; sums of some thousand terms round at 1e-13 of the norm
    scale = max(1.0, abs(lowest))
    assert abs(np.linalg.norm(x) - 1.0) < 1e-12
    assert np.linalg.norm(M @ x - E * x) < 1.1e-7
    assert abs(E - (x.conj() @ (M @ x)).real) < 1e-12 * scale
    assert abs(E - lowest) < 1e-12 * scale + 1e-10  # variance over the gaps here (above 1e-3)


@pytest.mark.parametrize("hop", [0.0, 1e-12j])
@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("levels", [1, 2, 4])
@pytest.mark.parametrize("nf,electrons", [(25, 2), (24, 3)])  # 300 and 2,024 rows
def test_few_distinct_values(api, nf, electrons, levels, seed, hop):
    """Densities whose sums over the electrons take one value, two (one orbital lies lower) or seven and
    ten (four levels); hop: a complex one of 1e-12, for complex vectors."""
    rng = np.random.default_rng(100 * seed + levels)
    c = 3.0 + 20.0 * rng.random()
    terms = sum((_number(api, i, c + 1.3 * (i % 4) if levels == 4 else c if levels == 1 or i else -c - 1.7)
                 for i in range(nf)), [])
    if hop:
        terms += [([0, 1 | api.CREATION], hop), ([1, 0 | api.CREATION], -hop)]
    H = api.Operator(nf, terms)
    b = _basis(api, nf, electrons)
    M = api.OperatorToDeterminantMatrix(H, b)
    X, E = api.EigensystemOnBasis(H, b, 1, {"Zero": 1e-14}, seed=seed)
    _check(M, X.cpu().numpy()[:, 0], E[0], np.linalg.eigvalsh(M)[0])


@pytest.mark.parametrize("inside,electrons", [(7, 3), (10, 2), (10, 3)])  # blocks of 35, 45 and 120 rows
def test_start_in_its_own_block(api, inside, electrons):
    """Hops among the first orbitals and among the others, no bridge: a start vector with all its
    electrons in the first ones reaches those rows only."""
    rng = np.random.default_rng(inside * electrons)
    nf = 24
    terms = sum((_number(api, i, -40.0 + rng.normal()) for i in range(nf)), [])
    for group in (range(inside), range(inside, nf)):
        for i in group:
            for j in group:
                if j < i:
                    v = float(rng.normal())
                    terms += [([i, j | api.CREATION], v), ([j, i | api.CREATION], v)]
    H = api.Operator(nf, terms)
    b = _basis(api, nf, electrons)
    M = api.OperatorToDeterminantMatrix(H, b)
    bits = np.unpackbits(b.dets_bytes(), axis=1)[:, :nf]
    rows = np.flatnonzero(bits[:, :inside].sum(axis=1) == electrons)
    assert not np.any(np.delete(M[rows], rows, axis=1))
    v = np.zeros((b.n, 1), dtype=complex)
    v[rows, 0] = rng.normal(size=len(rows))
    eng = api.engine()
    with eng.on_stream():
        x = eng.torch.from_numpy(v).cuda()
    en, it = np.zeros(1), C.c_int32()
    eng.check(eng.L.qg_block_groundstate(eng.ctx, H.handle(eng), b.h, 1, api._ptr(x), api._ptr(en), 1e-14, 400, 50,
                                         C.byref(it)))
    got = eng.to_host(x)[:, 0]
    assert not np.any(np.delete(got, rows))
    _check(M, got, en[0], np.linalg.eigvalsh(M[np.ix_(rows, rows)])[0])
