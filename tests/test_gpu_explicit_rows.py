"""One vector on a small basis through explicit rows: bitwise the list apply (which three passes of
one call run on, or a basis used fewer times), for complex vectors, real chains and pairs of
them, at the edges of slices (32 rows) and blocks (256); complex and sum operators stay on lists."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


def _basis(api, n):
    """n determinants of two electrons hopping on 40 orbitals, a diagonal and a few local terms."""
    rng = np.random.default_rng(n)
    nf = 40
    pairs = [(i, j) for i in range(nf) for j in range(i)]
    keep = [pairs[k] for k in rng.choice(len(pairs), n, replace=False)] if n < len(pairs) else pairs
    dets = ["".join("1" if o in p else "0" for o in range(nf)) for p in keep]
    terms = [([i, i | api.CREATION], float(rng.normal())) for i in range(nf)]
    for i in range(nf):
        for j in range(i):
            if rng.random() < 0.3:
                v = float(rng.normal())
                terms += [([i, j | api.CREATION], v), ([j, i | api.CREATION], v)]
    terms.append(([1, 0, 0x8002, 0x8003], 0.7))
    terms.append(([3, 2, 0x8000, 0x8001], 0.7))
    return api.Operator(nf, terms), api.Basis.from_bytes(nf, api.dets_to_bytes(dets, nf))[0]


def _apply(api, H, b, x):
    eng = api.engine()
    y = eng.empty(b.n)
    eng.check(eng.L.qg_apply(eng.ctx, H.handle(eng), b.h, b.h, api._ptr(x), api._ptr(y), 1))
    return eng.to_host(y)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 700, 780])
def test_apply_is_bitwise_the_list_apply(api, n):
    H, b = _basis(api, n)
    eng = api.engine()
    rng = np.random.default_rng(1)
    v = rng.normal(size=(b.n, 1)) + 1j * rng.normal(size=(b.n, 1))
    v[rng.integers(0, b.n)] = 0
    with eng.on_stream():
        x = eng.torch.from_numpy(v).cuda()
    got = [_apply(api, H, b, x) for _ in range(6)]  # lists, then rows from the fourth on
    assert all(np.array_equal(g, got[0]) for g in got)
    M = api.OperatorToDeterminantMatrix(H, b)
    assert np.abs(got[0] - M @ v).max() <= 1e-12 * max(1.0, np.abs(got[0]).max())


@pytest.mark.parametrize("kind", ["real", "pair", "complex"])
def test_chains_are_bitwise_those_of_lists(api, kind):
    """A long chain (rows) starts with the coefficients of a three-step one on a fresh basis (lists)."""
    from quanty_gb300 import workloads
    H, R, det, _ = workloads.anderson_impurity(nshell=3, hole_max=1, particle_max=1)
    eng = api.engine()
    rng = np.random.default_rng(2)
    out = []
    for ntri in (3, 12):
        b = api.closure(H, api.dets_to_bytes([det], H.nf), H.nf, R)
        if not out:
            cols = 2 if kind == "pair" else 1
            v = rng.normal(size=(b.n, cols)) + (1j * rng.normal(size=(b.n, cols)) if kind == "complex" else 0)
        with eng.on_stream():
            x = eng.torch.from_numpy(v.astype(complex)).cuda()
        out.append(api.lanczos_block(H, b, x, ntri, 1e-10, 0.5, eng))
    (a0, b0), (a1, b1) = out
    assert np.array_equal(a1[:, :4], a0[:, :4]) and np.array_equal(b1[:, :3], b0[:, :3])


def test_sum_operator_keeps_lists(api):
    """Values of a sum operator change between applies."""
    H, b = _basis(api, 300)
    S = api.OperatorSum([H, H], [1.0, 0.5])
    eng = api.engine()
    with eng.on_stream():
        x = eng.torch.ones((b.n, 1), dtype=eng.torch.complex128, device="cuda")
    for _ in range(5):
        y0 = _apply(api, S, b, x)
    S.set_coefficients([2.0, 1.0])
    assert np.abs(_apply(api, S, b, x) - 2 * y0).max() <= 1e-13 * np.abs(y0).max()
