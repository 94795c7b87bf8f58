"""Bases and operators shared by two contexts (streams): an operator of one context on a basis of
the other while both have work queued, against the results of one context with a wait after
every call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


@pytest.fixture()
def engines(api):
    a = api.engine()
    b = api.Engine(0)
    a.torch.cuda.set_stream(a.stream)
    yield a, b
    b.stream.synchronize()
    b.close()


def _operators(api, n):
    """Impurity Hamiltonians of one structure with different couplings, and a determinant."""
    from quanty_gb300 import workloads
    out = []
    for k in range(n):
        H, R, det, _ = workloads.anderson_impurity(nshell=3, hole_max=2, particle_max=1, udd=7.0 + 0.3 * k, field=0.1)
        out.append(H)
    return out, R, det


def _vectors(eng, n, count):
    rng = np.random.default_rng(n)
    with eng.on_stream():
        xs = [eng.torch.from_numpy(rng.normal(size=(n, 1)) + 1j * rng.normal(size=(n, 1))).cuda() for _ in range(count)]
    eng.torch.cuda.synchronize()
    return xs


def _apply(api, eng, h, b, x, y):
    eng.check(eng.L.qg_apply(eng.ctx, h, b.h, b.h, api._ptr(x), api._ptr(y), 1))


def _reference(api, eng, ops, b, xs):
    out = []
    for H in ops:
        for x in xs:
            y = eng.empty(b.n)
            _apply(api, eng, H.handle(eng), b, x, y)
            out.append(eng.to_host(y))
    return out


def test_operator_of_another_context(api, engines):
    """Handles of context A on a fresh basis of context B, whose moves are built while A has applies
    queued that take and return blocks of its own."""
    a, b = engines
    ops, R, det = _operators(api, 4)
    basis = {e: api.closure(ops[0], api.dets_to_bytes([det], ops[0].nf), ops[0].nf, R, -1, e) for e in (a, b)}
    xs = _vectors(a, basis[a].n, 2)
    want = _reference(api, a, ops, basis[a], xs)
    fresh = api.closure(ops[0], api.dets_to_bytes([det], ops[0].nf), ops[0].nf, R, -1, a)
    got = []
    for H in ops:
        for x in xs:
            ya, yb = a.empty(fresh.n), b.empty(fresh.n)
            a.torch.cuda.synchronize()  # the zeros of ya and yb
            _apply(api, a, H.handle(a), fresh, x, ya)
            _apply(api, b, H.handle(a), basis[b], x, yb)
            got.append((ya, yb))
    a.torch.cuda.synchronize()
    for w, (ya, yb) in zip(want, got):
        assert np.array_equal(w, ya.cpu().numpy()) and np.array_equal(w, yb.cpu().numpy())
