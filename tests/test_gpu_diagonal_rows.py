"""The diagonal of an operator on bases on both sides of the line between a warp and a thread per
row (16 rows per SM), with groups of one term and of many, real and complex values, one and two key
words, against the occupation numbers."""
import itertools

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
@pytest.mark.parametrize("nf", [33, 70])
@pytest.mark.parametrize("n", [1, 5, 33, 780, 0, 1000000])
def test_diagonal(api, n, nf, cplx):
    eng = api.engine()
    edge = 16 * eng.torch.cuda.get_device_properties(0).multi_processor_count
    n = {0: edge, 1000000: edge + 1}.get(n, n)
    rng = np.random.default_rng(n + nf)
    occ = np.zeros((n, nf), dtype=bool)
    for r, c in enumerate(itertools.islice(itertools.combinations(range(nf), 3), n)):
        occ[r, list(c)] = True
    val = lambda: complex(rng.normal(), rng.normal() if cplx and rng.random() < 0.5 else 0.0)  # noqa: E731
    terms, want, scale = [], np.zeros(n, dtype=complex), 0.0
    cre = api.CREATION
    for i in range(nf):
        for ops, f in (([i, i | cre], occ[:, i]), ([i | cre, i], ~occ[:, i])):  # an electron, a hole
            v = val()
            terms.append((ops, v))
            want += v * f
            scale += abs(v)
        for j in range(0, i, 3):
            v = val()
            terms.append(([i, i | cre, j, j | cre], v))
            want += v * (occ[:, i] & occ[:, j])
            scale += abs(v)
    H = api.Operator(nf, terms)
    dets = ["".join("1" if o else "0" for o in row) for row in occ]
    b, perm = api.Basis.from_bytes(nf, api.dets_to_bytes(dets, nf))
    index = {bytes(x): k for k, x in enumerate(api.dets_to_bytes(dets, nf))}
    order = [index[bytes(x)] for x in b.dets_bytes()]
    x = eng.empty(n)
    with eng.on_stream():
        x.fill_(1.0)
    y = eng.empty(n)
    eng.check(eng.L.qg_apply(eng.ctx, H.handle(eng), b.h, b.h, api._ptr(x), api._ptr(y), 1))
    got = eng.to_host(y)[:n, 0]
    # sums of at most len(terms) rounded additions, in another order
    assert np.abs(got - want[order]).max() <= len(terms) * 2.2e-16 * scale
