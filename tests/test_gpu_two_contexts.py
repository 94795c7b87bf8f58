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


def test_fresh_caches(api, engines):
    """Context B applies right behind A's call that built the moves, and right behind the one that built
    the explicit rows."""
    a, b = engines
    ops, R, det = _operators(api, 3)
    start = api.dets_to_bytes([det], ops[0].nf)
    basis = api.closure(ops[0], start, ops[0].nf, R, -1, a)
    xs = _vectors(a, basis.n, 2)
    want = _reference(api, a, ops, basis, xs)
    fresh = api.closure(ops[0], start, ops[0].nf, R, -1, a)
    ys = [[e.empty(fresh.n) for _ in range(6)] for e in (a, b)]
    a.torch.cuda.synchronize()
    for i, H in enumerate(ops):
        for k in range(6):  # the rows are there from the fourth apply on; B alone applies on the odd rounds
            x = xs[k % 2]
            if (i + k) % 2 == 0:
                _apply(api, a, H.handle(a), fresh, x, ys[0][k])
            _apply(api, b, H.handle(a), fresh, x, ys[1][k])
        a.torch.cuda.synchronize()
        for k in range(6):
            w = want[2 * i + k % 2]
            assert np.array_equal(w, ys[1][k].cpu().numpy())
            assert (i + k) % 2 or np.array_equal(w, ys[0][k].cpu().numpy())


def test_evicted_caches(api, engines):
    """A basis keeps four operators: context A goes round seven of them, so that caches are dropped and
    their blocks used again, while context B has applies queued on them."""
    a, b = engines
    ops, R, det = _operators(api, 7)
    basis = api.closure(ops[0], api.dets_to_bytes([det], ops[0].nf), ops[0].nf, R, -1, a)
    xs = _vectors(a, basis.n, 1)
    want = _reference(api, a, ops, basis, xs)
    ys = [b.empty(basis.n) for _ in range(14)]
    ya = a.empty(basis.n)
    val = np.zeros(2)
    a.torch.cuda.synchronize()
    for k in range(14):
        h = ops[k % 7].handle(a)
        for _ in range(8):
            _apply(api, b, h, basis, xs[0], ys[k])
        # another operator: a new cache, an eviction from the fifth on; and blocks taken and written
        _apply(api, a, ops[(k + 1) % 7].handle(a), basis, xs[0], ya)
        a.check(a.L.qg_expectation(a.ctx, ops[(k + 1) % 7].handle(a), basis.h, api._ptr(xs[0]), 1, api._ptr(val)))
    a.torch.cuda.synchronize()
    assert all(np.array_equal(want[k % 7], ys[k].cpu().numpy()) for k in range(14))
