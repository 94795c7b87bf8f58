"""Device memory kept by a context: results do not depend on it (several threads with a context
each, alternating sizes so that blocks are reused), it is bounded, and qg_finalize gives it back."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from quanty_gb300 import build
    build.build()
    from quanty_gb300 import api
    return api


def _states(api, H, eng):
    out = []
    from quanty_gb300 import workloads
    for nshell, holes, particles in ((0, 0, 0), (1, 0, 1), (2, 1, 1), (1, 0, 2)):
        Hn, R, det, _ = workloads.anderson_impurity(nshell=nshell, hole_max=holes, particle_max=particles)
        b = api.closure(Hn, api.dets_to_bytes([det], Hn.nf), Hn.nf, R, -1, eng)
        v = np.random.default_rng(b.n).normal(size=b.n) + 0j
        out.append((Hn, api.Wavefunction(Hn.nf, b.dets_bytes(), v)))
    return out


def _run(api, work, eng, order):
    got = {}
    for i in order:
        Hn, psi = work[i]
        r = api.OperatorPsi(Hn, psi, eng=eng)
        got.setdefault(i, []).append((r.det.tobytes(), r.val.tobytes(), api.PsiOperatorPsi(Hn, psi, eng)))
    return got


def test_threads_and_reuse(api):
    eng0 = api.engine()
    work = _states(api, None, eng0)
    want = _run(api, work, eng0, range(len(work)))
    results, errors = [], []

    def worker(seed):
        try:
            eng = api.Engine(0)
            order = list(np.random.default_rng(seed).integers(0, len(work), 24))
            results.append(_run(api, work, eng, order))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=worker, args=(s,)) for s in range(3)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors
    for got in results:
        for i, rs in got.items():
            assert all(r == want[i][0] for r in rs)


def test_bounded_and_given_back(api):
    import gc
    torch = api.engine().torch
    torch.cuda.synchronize()
    gc.collect()
    before = torch.cuda.mem_get_info()[0]
    eng = api.Engine(0)
    work = _states(api, None, eng)
    _run(api, work, eng, [3, 2, 3, 1])
    del work
    gc.collect()
    eng.stream.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    assert held < (1 << 30) + (256 << 20)  # the bound, and what the driver and torch keep
    eng.close()
    torch.cuda.set_stream(api.engine().stream)
    torch.cuda.empty_cache()
    assert before - torch.cuda.mem_get_info()[0] < (256 << 20)
