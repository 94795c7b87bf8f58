"""Both forms of the list kernel (more resident blocks, or more registers) around the lines between
them: two, six and eight blocks of 256 rows per SM (77,824, 233,472 and 311,296 rows on 152 SMs).
The first apply goes by the rule, the second times both, later ones use what was faster; every
vector's bits are those of the vector alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


def _apply(api, H, b, x):
    eng = api.engine()
    y = eng.empty(b.n, x.shape[1])
    eng.check(eng.L.qg_apply(eng.ctx, H.handle(eng), b.h, b.h, api._ptr(x), api._ptr(y), x.shape[1]))
    return y


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("nshell,holes,particles", [(2, 1, 2), (6, 0, 2), (3, 1, 2), (2, 2, 2), (4, 1, 2)])
def test_bitwise_the_vector_alone(api, nshell, holes, particles, cplx):
    from quanty_gb300 import workloads
    H, R, det, _ = workloads.anderson_impurity(nshell=nshell, hole_max=holes, particle_max=particles, field=0.1,
                                               complex_field=cplx)
    b = api.closure(H, api.dets_to_bytes([det], H.nf), H.nf, R)
    eng = api.engine()
    rng = np.random.default_rng(b.n)
    v = rng.normal(size=(b.n, 11)) + 1j * rng.normal(size=(b.n, 11))
    with eng.on_stream():
        x = eng.torch.from_numpy(v).cuda()
        alone = eng.torch.cat([_apply(api, H, b, x[:, k:k + 1].contiguous()) for k in range(11)], 1)
        for nvec in (2, 3, 4, 8, 11):
            part = x[:, :nvec].contiguous()
            for _ in range(3):
                assert eng.torch.equal(_apply(api, H, b, part), alone[:, :nvec])
    # <v|H v> from another call
    w = api.Wavefunction(H.nf, b.dets_bytes(), v[:, 0])
    e = api.PsiOperatorPsi(H, w)
    y = eng.to_host(alone[:, :1])[:, 0]
    # sums of some 1e5 products of size |v|^2 |H|, each rounded
    assert abs(np.vdot(v[:, 0], y) - e) <= 1e-12 * np.linalg.norm(v[:, 0]) * np.linalg.norm(y)
