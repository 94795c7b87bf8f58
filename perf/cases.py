"""The work whose speed this library is judged by: calls through its public entry points, over the
sizes, data types and options its users bring.

A case is one call (or the short sequence a program makes of it) on a discretised-bath Anderson
impurity of ``quanty_gb300.workloads`` (16 + 10 * shells spin-orbitals), on the 16-orbital ion or on
the 26-orbital ligand-field ion.  The kinds:

* ``psi``      ``OperatorPsi``: H|psi> or T|psi> with basis growth, a wavefunction on the host in and
               out, as a script writes ``O * psi``;
* ``apply``    ``qg_apply``: H on device vectors of a closed basis, the product every solver repeats;
* ``host``     ``qg_apply_host``: the same on page-locked host vectors, the reference's convention;
* ``lanczos``  ``lanczos_block``: the tridiagonal coefficients of one or more chains;
* ``spectra``  ``CreateSpectra`` on the ligand-field ion, host states in, spectra out;
* ``dense``    ``CreateSpectra`` below DenseBorder: the dense branch, poles and spectra out;
* ``ground``   ``EigensystemOnBasis`` and ``CreateSpectraResident``: the ground state, then its spectra;
* ``rixs``     ``CreateResonantSpectra``, Krylov branch.

Recursions without reorthogonalisation are run for as many steps as their coefficients are set by
their input (24 here); past the loss of orthogonality rounding alone decides them.  Eigenvectors are
fixed up to a phase only, so the ``ground`` and ``dense`` cases return what a program computes from
them (energies, poles, spectra).  ``exact`` restates every computed result in plain torch, in
64-bit numbers.
"""
import itertools
import math

import numpy as np
import torch

from quanty_gb300 import api, workloads

NTRI = 24       # steps of a Lanczos chain
GAMMA = 0.5     # eV, the broadening of the spectra
FIELD = 0.1     # eV, the exchange field of a magnet, which splits its ground multiplet
ZERO = 1e-12    # eV^2, the variance of states that spectra are built on


def listed():
    return [
        # T|psi> of an isolated ion, 45 determinants: the smallest call a script makes, all latency
        {"name": "psi_ion", "kind": "psi", "shells": 0, "bath": 0, "holes": 0, "particles": 0, "operator": "Tz"},
        # H|psi> grown out of an odd-sized host wavefunction of a 46-orbital impurity
        {"name": "psi_46", "kind": "psi", "shells": 3, "bath": 0, "holes": 3, "particles": 1, "operator": "H"},
        # a small complex Hamiltonian (spin-orbit or magnetic field along a general axis), one vector
        {"name": "apply_36_complex", "kind": "apply", "shells": 2, "bath": 0, "holes": 2, "particles": 2, "core": 0,
         "complex": True, "vectors": 1},
        # sixteen thermal states at once on the core-excited basis of a 66-orbital impurity
        {"name": "apply_66_block", "kind": "apply", "shells": 5, "bath": 0, "holes": 1, "particles": 2, "core": 1,
         "complex": False, "vectors": 16},
        # the largest configuration of the benchmark: 47,481,880 determinants
        {"name": "apply_86", "kind": "apply", "shells": 7, "bath": 0, "holes": 3, "particles": 2, "core": 0,
         "complex": False, "vectors": 1},
        # a caller that keeps its vectors in page-locked host memory
        {"name": "host_76", "kind": "host", "shells": 6, "bath": 0, "holes": 2, "particles": 2, "core": 0,
         "complex": False, "vectors": 1},
        # one real chain (a real ground state of a real Hamiltonian) on 3,899,040 determinants
        {"name": "lanczos_76_real", "kind": "lanczos", "shells": 6, "bath": 0, "holes": 1, "particles": 2, "core": 1,
         "complex": False, "vectors": 1, "real": True},
        # polarisations x states as one multi-vector recursion, complex start vectors
        {"name": "lanczos_56_block", "kind": "lanczos", "shells": 4, "bath": 0, "holes": 1, "particles": 2, "core": 1,
         "complex": False, "vectors": 6, "real": False},
        # XAS of the ligand-field ion: three states, three polarisations, the reference's tutorial size
        {"name": "spectra_26", "kind": "spectra", "states": 3, "operators": 3, "ne": 2048},
        # a basis below DenseBorder, where CreateSpectra diagonalises
        {"name": "dense_56", "kind": "dense", "shells": 4, "bath": 0, "holes": 2, "particles": 0, "vectors": 2, "ne": 1000},
        # the ground state and its XAS, the whole calculation on the device
        {"name": "ground_46", "kind": "ground", "shells": 3, "bath": 0, "holes": 2, "particles": 1, "ne": 2048},
        # RIXS: sixteen incident energies, three emission polarisations
        {"name": "rixs_46", "kind": "rixs", "shells": 3, "bath": 0, "holes": 1, "particles": 2, "ne1": 15, "ne2": 512},
    ]


# the largest basis a drawn case of each kind may have (times its vectors for the multi-vector kinds)
LIMIT = {"psi": 40000, "apply": 47.5e6, "host": 10.4e6, "lanczos": 3.9e6, "dense": 800, "ground": 30000,
         "rixs": 130000}


def draw(rng):
    kind = rng.choice(("psi", "apply", "apply", "host", "lanczos", "lanczos", "spectra", "dense", "ground", "rixs"))
    if kind == "spectra":
        return {"kind": kind, "states": rng.randint(1, 4), "operators": rng.randint(1, 3),
                "ne": int(math.exp(rng.uniform(math.log(300), math.log(2600))))}
    while True:
        c = {"kind": kind, "shells": rng.randint(1, 7), "bath": rng.randint(0, 9999),
             "holes": rng.randint(0, 3), "particles": rng.randint(0, 2)}
        if kind in ("apply", "host", "lanczos"):
            c["core"] = rng.randint(0, 1)
            c["complex"] = rng.random() < 0.25
            c["vectors"] = 1 if kind == "host" or rng.random() < 0.5 else rng.randint(2, 24 if kind == "apply" else 8)
        if kind == "psi":
            c["operator"] = rng.choice(("H", "Tx", "Tz"))
        if kind == "lanczos":
            c["real"] = not c["complex"] and rng.random() < 0.5
        if kind == "ground":
            c["ne"] = rng.randint(500, 2500)
        if kind == "dense":
            c["vectors"] = rng.randint(1, 3)
            c["ne"] = rng.randint(500, 2000)
        if kind == "rixs":
            c["ne1"], c["ne2"] = rng.randint(3, 15), rng.randint(200, 600)
        n = _size(c, 1 if kind in ("ground", "rixs") else c.get("core", 0))
        low = {"psi": 40, "dense": 100, "ground": 9000, "rixs": 9000}.get(kind, 3000 if kind != "lanczos" else 9000)
        # sizes spread over their logarithm: large ones are thinned out, small ones mostly refused
        cost = n * (max(1, c["vectors"] * 0.7) if kind in ("apply", "lanczos") else 1)
        if kind in ("ground", "rixs"):
            cost = _size(c, 0)
        if low <= n and cost <= LIMIT[kind]:
            return c


# ----------------------------------------------------------------------------- the material

def _material(c, core=None):
    """H, the occupation windows, the seed determinant and the bath of a case."""
    core = c.get("core", 0) if core is None else core
    H, R, seed, info = workloads.anderson_impurity(
        nshell=c["shells"], seed=c["bath"], hole_max=c["holes"], particle_max=c["particles"], core_holes=core,
        complex_field=bool(c.get("complex")), field=FIELD if c["kind"] == "ground" else 0.01)
    if core:  # one 2p electron lifted into the 3d shell
        s = list(seed)
        s[0], s[s.index("0", 6, 16)] = "0", "1"
        seed = "".join(s)
    return H, R, seed, info


def _filled(c):
    eps = np.sort(np.random.default_rng(c["bath"]).uniform(-5.0, 5.0, c["shells"]))
    f = int((eps < 0).sum())
    return f, c["shells"] - f


def _size(c, core):
    f, e = _filled(c)
    return (6 if core else 1) * workloads.sector_size(f, e, nd0=9 if core else 8, hole_max=c["holes"],
                                                      particle_max=c["particles"])


def _dipole(nf, name):
    return api.Operator(nf, workloads.atomic()[name].terms, name=name)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (int(seed) % (1 << 31)) + 17)
    return g


def _vectors(n, k, seed, real):
    """Normalised vectors whose amplitudes spread over several decades, as those of a state do."""
    g = _gen(seed)
    x = torch.randn((n, k), dtype=torch.float64, device="cuda", generator=g).to(torch.complex128)
    if not real:
        x += 1j * torch.randn((n, k), dtype=torch.float64, device="cuda", generator=g)
    x *= torch.pow(10.0, -3.0 * torch.rand((n, 1), dtype=torch.float64, device="cuda", generator=g))
    return (x / torch.linalg.vector_norm(x, dim=0, keepdim=True)).contiguous()


def _local_operators(c, count, seed):
    """Hermitian one-body operators on the 3d shell (a spin, an orbital moment, a field): seeded."""
    rng = np.random.default_rng(int(seed) + 5)
    out = []
    for _ in range(count):
        terms = []
        for a in range(6, 16):
            for b in range(a, 16):
                v = complex(rng.normal(), rng.normal() if a != b else 0.0)
                terms.append(([b, a | api.CREATION], v))
                if a != b:
                    terms.append(([a, b | api.CREATION], v.conjugate()))
        out.append(api.Operator(16 + 10 * c["shells"], terms))
    return out


def prepare(case, seed):
    c, kind = case, case["kind"]
    eng = api.engine()
    s = {"case": c, "eng": eng}
    if kind == "spectra":
        ops, R = workloads.ligand_field()
        dets = api.enumerate_restricted(26, R)
        rng = np.random.default_rng(int(seed))
        s["H"], s["T"] = ops["HX"], [ops[k] for k in ("Tx", "Ty", "Tz")[:c["operators"]]]
        s["psi"] = []
        for _ in range(c["states"]):
            v = rng.standard_normal(len(dets)) * 10.0 ** (-3.0 * rng.random(len(dets)))
            s["psi"].append(api.Wavefunction(26, dets, v / np.linalg.norm(v)))
        s["options"] = {"Method": "Lanczos", "NTri": 200, "NE": c["ne"], "Emin": -10.0, "Emax": 20.0, "Gamma": GAMMA}
        return s
    H, R, det, _ = _material(c)
    s["H"], nf = H, H.nf
    if kind == "psi":
        b = api.closure(H, api.dets_to_bytes([det], nf), nf, R, -1, eng)
        v = _vectors(b.n, 1, seed, False)[:, 0].cpu().numpy()
        s["psi"] = api.Wavefunction(nf, b.dets_bytes(), v)
        s["O"] = H if c["operator"] == "H" else _dipole(nf, c["operator"])
        return s
    b = s["basis"] = api.closure(H, api.dets_to_bytes([det], nf), nf, R, -1, eng)
    if kind in ("apply", "lanczos"):
        s["x"] = _vectors(b.n, c["vectors"], seed, bool(c.get("real")))
        s["y"] = torch.empty_like(s["x"])
    elif kind == "host":
        x = _vectors(b.n, 1, seed, False)
        s["x"] = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
        s["x"].copy_(x)
        s["y"] = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
    elif kind == "dense":
        rng = np.random.default_rng(int(seed))
        v = rng.standard_normal(b.n) * 10.0 ** (-3.0 * rng.random(b.n))
        s["psi"] = api.Wavefunction(nf, b.dets_bytes(), v / np.linalg.norm(v))
        s["T"] = _local_operators(c, c["vectors"], seed)
        s["options"] = {"NE": c["ne"], "Emin": -30.0, "Emax": 30.0, "Gamma": GAMMA, "Restrictions": R}
    elif kind == "ground":
        s["T"] = [_dipole(nf, k) for k in ("Tx", "Tz")]
        s["seed"] = 1 + int(seed) % (1 << 30)
        s["options"] = {"NTri": NTRI, "NE": c["ne"], "Emin": -20.0, "Emax": 20.0, "Gamma": GAMMA,
                        "Restrictions": _material(c, 1)[1]}
    elif kind == "rixs":
        v = _vectors(b.n, 1, seed, True)[:, 0].cpu().numpy()
        s["psi"] = api.Wavefunction(nf, b.dets_bytes(), v)
        s["T1"] = _dipole(nf, "Tz")
        s["T2"] = [_dipole(nf, k).dagger() for k in ("Tx", "Ty", "Tz")]
        s["options"] = _rixs_options(c)
    return s


def _rixs_options(c):
    return {"NTri1": NTRI, "NTri2": NTRI, "Emin1": -8.0, "Emax1": 8.0, "NE1": c["ne1"], "Gamma1": 0.4,
            "Emin2": -2.0, "Emax2": 10.0, "NE2": c["ne2"], "Gamma2": GAMMA,
            "Restrictions1": _material(c, 1)[1], "Restrictions2": _material(c, 0)[1]}


def run(state):
    s, kind, eng = state, state["case"]["kind"], state["eng"]
    if kind == "psi":
        out = api.OperatorPsi(s["O"], s["psi"])
        return {"det": out.det, "val": out.val}
    if kind == "apply":
        H, b, x, y = s["H"], s["basis"], s["x"], s["y"]
        eng.check(eng.L.qg_apply(eng.ctx, H.handle(eng), b.h, b.h, api._ptr(x), api._ptr(y), x.shape[1]))
        return y
    if kind == "host":
        H, b, x, y = s["H"], s["basis"], s["x"], s["y"]
        eng.check(eng.L.qg_apply_host(eng.ctx, H.handle(eng), b.h, b.h, api._ptr(x), api._ptr(y), 1))
        return y
    if kind == "lanczos":
        a, b = api.lanczos_block(s["H"], s["basis"], s["x"], NTRI, api.DEFAULTS["Epsilon"], GAMMA, eng)
        return {"a": a, "b": b}
    if kind == "spectra":
        return api.CreateSpectra(s["H"], s["T"], s["psi"], s["options"], eng)[0].G
    if kind == "dense":
        S, poles = api.CreateSpectra(s["H"], s["T"], s["psi"], s["options"], eng)
        return {"G": S.G, "poles": [p[0] for p in poles]}
    if kind == "ground":
        X, E = api.EigensystemOnBasis(s["H"], s["basis"], 1, {"Zero": ZERO}, eng, seed=s["seed"])
        S = api.CreateSpectraResident(s["H"], s["T"], s["basis"], X, E, s["options"], eng)[0]
        return {"E": E, "G": S.G}
    G, _ = api.CreateResonantSpectra(s["H"], s["H"], s["T1"], s["T2"], s["psi"], s["options"], eng)
    return G


# ----------------------------------------------------------------------------- the least work

def _connections(c, core):
    """Connections per determinant that stay inside the windows (off the diagonal, and all of
    them), from 256 determinants of the sector drawn on the host."""
    H, R, _, info = _material(c, core)
    rng = np.random.default_rng(3)
    f = info["filled_shells"]
    e = [k for k in range(c["shells"]) if k not in f]
    full = sum(1 << i for i in range(6 - core)) << core
    windows = [(sum(1 << i for i, ch in enumerate(m) if ch == "1"), lo, hi) for m, lo, hi in R]
    shell = lambda ks: [o for k in ks for o in range(16 + 10 * k, 26 + 10 * k)]  # noqa: E731
    classes, weight = [], []
    for h in range(c["holes"] + 1):
        for p in range(c["particles"] + 1):
            nd = 8 + core + h - p
            if 0 <= nd <= 10 and (h == 0 or f) and (p == 0 or e):
                classes.append((h, p, nd))
                weight.append(math.comb(10 * len(f), h) * math.comb(10 * len(e), p) * math.comb(10, nd))
    weight = np.array(weight, dtype=float) / sum(weight)
    off = 0
    terms = [(ops, v) for ops, v in H.terms if v != 0]
    dets = []
    while len(dets) < 256:
        h, p, nd = classes[rng.choice(len(classes), p=weight)]
        d = full | sum(1 << int(i) for i in rng.choice(range(6, 16), nd, replace=False))
        d |= sum(1 << o for o in shell(f))
        if h:
            d &= ~sum(1 << int(i) for i in rng.choice(shell(f), h, replace=False))
        if p:
            d |= sum(1 << int(i) for i in rng.choice(shell(e), p, replace=False))
        if all(lo <= (d & m).bit_count() <= hi for m, lo, hi in windows):
            dets.append(d)
    for d in dets:
        reached = set()
        for ops, _ in terms:
            t = d
            for o in ops:
                bit = 1 << (o & 0x7FFF)
                if bool(t & bit) == bool(o & 0x8000):
                    t = -1
                    break
                t ^= bit
            if t >= 0 and t != d and all(lo <= (t & m).bit_count() <= hi for m, lo, hi in windows):
                reached.add(t)
        off += len(reached)
    return off / len(dets)


def work(case):
    """Bytes: keys, input and output vectors once.  Operations: a multiply and an add per real
    product of every distinct connection and of the diagonal."""
    c, kind = case, case["kind"]
    if kind == "spectra":
        pairs = c["states"] * c["operators"]
        return {"bytes": 190 * 20 * c["states"] + pairs * c["ne"] * 16,
                "flops": pairs * (200 * 120 * 12 * 4 + c["ne"] * 200 * 14)}
    n = _size(c, c.get("core", 0))
    key = 8 * (2 if c["shells"] > 4 else 1)
    if kind == "dense":
        return {"bytes": n * (key + 16) + c["vectors"] * c["ne"] * 16, "flops": 4 / 3 * n ** 3 + c["ne"] * c["vectors"] * n * 8}
    if kind == "psi":
        if c["operator"] != "H":
            return {"bytes": 2 * n * (key + 16), "flops": n * 30 * 4}
        k = _connections(c, 0)
        return {"bytes": n * (key + 16) * 2, "flops": n * (k + 1) * 4}
    per = 2 if c.get("real") or kind in ("ground", "rixs") else 8 if c.get("complex") else 4
    amp = 8 if c.get("real") else 16
    if kind in ("apply", "host"):
        k = _connections(c, c["core"])
        return {"bytes": n * (key + 2 * amp * c["vectors"]), "flops": n * (k + 1) * per * c["vectors"]}
    if kind == "lanczos":
        k = _connections(c, c["core"])
        return {"bytes": NTRI * n * (key + 3 * amp * c["vectors"]), "flops": NTRI * n * (k + 4) * per * c["vectors"]}
    n1, k1 = _size(c, 1), _connections(c, 1)
    if kind == "ground":
        return {"bytes": NTRI * (n + n1) * (key + 24),
                "flops": (NTRI * n1 * (k1 + 4) * 2 + 150 * n * (k1 + 4) + 2 * 150 ** 2 * n) * 2}
    v = 3 * (c["ne1"] + 1)
    return {"bytes": NTRI * (n1 * 24 + n * (key + 3 * 16 * v)),
            "flops": NTRI * n1 * (k1 + 2 * NTRI) * 2 + NTRI * n * (k1 + 4) * v * 4}


# ----------------------------------------------------------------------------- the same in plain torch


def _pair(orbitals):
    """Orbitals as (hi, lo): orbital i < 62 is bit 61 - i of hi, the others bit 123 - i of lo, so the
    order of (hi, lo) is the order of the determinants' strings."""
    hi = sum(1 << (61 - i) for i in orbitals if i < 62)
    return hi, sum(1 << (123 - i) for i in orbitals if i >= 62)


def _plain_device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _sorted_pairs(hi, lo):
    o = torch.sort(lo, stable=True)[1]
    o = o[torch.sort(hi[o], stable=True)[1]]
    return hi[o], lo[o]


def _sector(c, core):
    """Every determinant of the sector, sorted."""
    _, _, _, info = _material(c, core)
    f = info["filled_shells"]
    e = [k for k in range(c["shells"]) if k not in f]
    dev = _plain_device()
    fo = [o for k in f for o in range(16 + 10 * k, 26 + 10 * k)]
    eo = [o for k in e for o in range(16 + 10 * k, 26 + 10 * k)]

    def sets(orbs, m):
        for t in itertools.combinations(orbs, m):
            shells = [(o - 16) // 10 for o in t]
            if all(shells.count(k) <= 2 for k in shells):
                yield t

    def words(rows):
        return torch.tensor([_pair(r) for r in rows], dtype=torch.int64, device=dev).reshape(-1, 2)

    core_sets = [tuple(range(6))] if not core else list(itertools.combinations(range(6), 5))
    his, los = [], []
    base = _pair(fo)
    for h in range(c["holes"] + 1):
        hs = words(sets(fo, h)) if h else words([()])
        if not len(hs):
            continue
        hs = torch.tensor(base, dtype=torch.int64, device=dev)[None, :] ^ hs
        for p in range(c["particles"] + 1):
            nd = 8 + core + h - p
            ps = words(sets(eo, p)) if p else words([()])
            if not 0 <= nd <= 10 or not len(ps):
                continue
            bath = (hs[:, None, :] | ps[None, :, :]).reshape(-1, 2)
            for cs in core_sets:
                imp = words([cs + t for t in itertools.combinations(range(6, 16), nd)])
                his.append((imp[:, None, 0] | bath[None, :, 0]).reshape(-1))
                los.append(bath[None, :, 1].expand(len(imp), -1).reshape(-1))
    return _sorted_pairs(torch.cat(his), torch.cat(los))


def _hash(hi, lo):
    x = hi * -7046029254386353131
    x = ((x ^ (x >> 31)) + lo) * -2960836687038522477
    return (x ^ (x >> 29)) * -7046029254386353131


class _Lookup:
    def __init__(self, hi, lo):
        self.hi, self.lo = hi, lo
        self.h, self.row = torch.sort(_hash(hi, lo))
        if len(hi) > 1 and bool((self.h[1:] == self.h[:-1]).any()):
            raise RuntimeError("two determinants share a hash")

    def __call__(self, hi, lo):
        """Rows of the given determinants, and which of them are there."""
        p = torch.searchsorted(self.h, _hash(hi, lo)).clamp_(max=len(self.h) - 1)
        r = self.row[p]
        return r, (self.hi[r] == hi) & (self.lo[r] == lo)


def _term(ops, hi, lo):
    """The rows a ladder string applies to, their targets and signs (+1, -1)."""
    want, state = {}, {}
    for o in ops:
        i, create = o & 0x7FFF, bool(o & 0x8000)
        if i in state:
            if state[i] == create:
                return None
        else:
            want[i] = not create
        state[i] = create
    n1, n0 = _pair([i for i in want if want[i]]), _pair([i for i in want if not want[i]])
    ok = ((hi & (n1[0] | n0[0])) == n1[0]) & ((lo & (n1[1] | n0[1])) == n1[1])
    rows = torch.nonzero(ok).reshape(-1)
    th, tl = hi[rows], lo[rows]
    par = torch.zeros_like(rows)
    for o in ops:
        i = o & 0x7FFF
        mh, ml = _pair(range(i))
        x = (th & mh) ^ (tl & ml)
        for k in (32, 16, 8, 4, 2, 1):
            x = x ^ (x >> k)
        par ^= x & 1
        fh, fl = _pair([i])
        th, tl = th ^ fh, tl ^ fl
    return rows, th, tl, 1.0 - 2.0 * par.to(torch.float64)


def _push(O, hi, lo, look, x, n_out):
    """O x from the determinants (hi, lo) into those of `look` (complex columns)."""
    y = torch.zeros((n_out, x.shape[1]), dtype=torch.complex128, device=x.device)
    for ops, v in O.terms:
        got = _term(ops, hi, lo) if v != 0 else None
        if got is None or not len(got[0]):
            continue
        rows, th, tl, sign = got
        to, there = look(th, tl)
        if not bool(there.all()):
            rows, to, sign = rows[there], to[there], sign[there]
        y[to] += (v * sign)[:, None] * x[rows]  # a string takes no two determinants to one
    return y


def _matrix(H, hi, lo):
    """H on the sector as a sparse matrix: a function that applies it to complex columns."""
    look, n = _Lookup(hi, lo), len(hi)
    real = all(v.imag == 0 for _, v in H.terms)
    to, frm, val = [], [], []
    for ops, v in H.terms:
        got = _term(ops, hi, lo) if v != 0 else None
        if got is None or not len(got[0]):
            continue
        rows, th, tl, sign = got
        t, there = look(th, tl)
        to.append(t[there])
        frm.append(rows[there])
        val.append((v.real if real else v) * sign[there])
    to, frm, val = torch.cat(to), torch.cat(frm), torch.cat(val)
    key, o = torch.sort(to * n + frm)
    del to, frm
    uniq, inv = torch.unique_consecutive(key, return_inverse=True)
    v = torch.zeros(len(uniq), dtype=val.dtype, device=val.device)
    v.index_add_(0, inv, val[o])
    row, col = uniq // n, uniq % n
    start = torch.searchsorted(row, torch.arange(n + 1, device=row.device))
    M = torch.sparse_csr_tensor(start, col, v, (n, n))

    def times(x):
        if not real:
            return M @ x
        z = torch.view_as_real(x.contiguous()).reshape(n, -1)
        return torch.view_as_complex((M @ z).reshape(n, -1, 2).contiguous())
    return times


def _plain_lanczos(times, x, ntri, eps, gamma):
    """Three-term recursion of every column: a (columns, ntri + 1), b (columns, ntri)."""
    k = x.shape[1]
    a = torch.zeros((k, ntri + 1), dtype=torch.float64, device=x.device)
    b = torch.zeros((k, ntri), dtype=torch.float64, device=x.device)
    err = torch.ones(k, dtype=torch.float64, device=x.device)
    prev, w = None, x
    for i in range(ntri):
        if i:
            w = w - a[:, i] * v
        b[:, i] = torch.linalg.vector_norm(w, dim=0)
        new = w / b[:, i]
        new = torch.where(new.abs() > eps / err, new, torch.zeros_like(new))
        if i:
            prev = v
            err = err * b[:, i] ** 2 / (b[:, i] ** 2 + 4 * gamma ** 2)
        v = new
        w = times(v)
        a[:, i + 1] = (v.conj() * w).sum(0).real
        if i:
            w = w - b[:, i] * prev
    return a, b


def _fraction(a, b, w, gamma):
    """The continued fraction of every row of (a, b) at the frequencies of the same row of w."""
    g = torch.zeros(w.shape, dtype=torch.complex128, device=w.device)
    z = w + 0.5j * gamma
    for k in range(b.shape[1] - 1, -1, -1):
        g = b[:, k:k + 1] ** 2 / (z - a[:, k + 1:k + 2] - g)
    return g


def _grid(emin, emax, ne, dev):
    return emin + torch.arange(ne + 1, dtype=torch.float64, device=dev) * ((emax - emin) / ne)


def _bytes_of(hi, lo, nf):
    out = np.zeros((len(hi), (nf + 7) // 8), dtype=np.uint8)
    h, l = hi.cpu().numpy(), lo.cpu().numpy()
    for i in range(nf):
        bit = (h >> (61 - i)) & 1 if i < 62 else (l >> (123 - i)) & 1
        out[:, i >> 3] |= (bit << (7 - (i & 7))).astype(np.uint8)
    return out


def _pairs_of(det, nf):
    bits = np.unpackbits(det, axis=1)[:, :nf].astype(np.int64)
    hi, lo = np.zeros(len(det), dtype=np.int64), np.zeros(len(det), dtype=np.int64)
    for i in range(nf):
        if i < 62:
            hi |= bits[:, i] << (61 - i)
        else:
            lo |= bits[:, i] << (123 - i)
    dev = _plain_device()
    return torch.from_numpy(hi).to(dev), torch.from_numpy(lo).to(dev)


def _grown(O, hi, lo):
    """The determinants O reaches, sorted."""
    hs, ls = [], []
    for ops, v in O.terms:
        got = _term(ops, hi, lo) if v != 0 else None
        if got is not None and len(got[0]):
            hs.append(got[1])
            ls.append(got[2])
    both = torch.unique(torch.stack([torch.cat(hs), torch.cat(ls)], dim=1), dim=0)
    return both[:, 0].contiguous(), both[:, 1].contiguous()


def _expect(times, x):
    return (x.conj() * times(x)).sum(0).real


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "spectra":
        return _exact_spectra(c, seed)
    dev = _plain_device()
    H = _material(c)[0]
    nf = H.nf
    eps = float(np.sqrt(np.finfo(float).eps)) / 100
    hi, lo = _sector(c, c.get("core", 0))
    n = len(hi)
    if kind in ("apply", "host"):
        x = _vectors(n, c["vectors"], seed, False)
        y = _push(H, hi, lo, _Lookup(hi, lo), x, n)
        return y.cpu() if kind == "host" else y
    if kind == "psi":
        O = H if c["operator"] == "H" else _dipole(nf, c["operator"])
        th, tl = _grown(O, hi, lo)
        y = _push(O, hi, lo, _Lookup(th, tl), _vectors(n, 1, seed, False), len(th))
        return {"det": _bytes_of(th, tl, nf), "val": y[:, 0].cpu().numpy()}
    if kind == "lanczos":
        a, b = _plain_lanczos(_matrix(H, hi, lo), _vectors(n, c["vectors"], seed, bool(c["real"])), NTRI, eps, GAMMA)
        return {"a": a.cpu().numpy(), "b": b.cpu().numpy()}
    if kind == "dense":
        times = _matrix(H, hi, lo)
        M = times(torch.eye(n, dtype=torch.complex128, device=dev))
        w, V = torch.linalg.eigh((M + M.conj().T) / 2)
        rng = np.random.default_rng(int(seed))
        v = rng.standard_normal(n) * 10.0 ** (-3.0 * rng.random(n))
        x = torch.from_numpy(v / np.linalg.norm(v)).to(dev).to(torch.complex128)[:, None]
        e0 = float(_expect(times, x)[0])
        look = _Lookup(hi, lo)
        om = _grid(-30.0, 30.0, c["ne"], dev) + e0 + 0.5j * GAMMA
        G = []
        for T in _local_operators(c, c["vectors"], seed):
            wt = (V.conj().T @ _push(T, hi, lo, look, x, n))[:, 0].abs() ** 2
            G.append((wt[None, :] / (om[:, None] - w[None, :])).sum(1))
        return {"G": torch.stack(G).cpu().numpy(), "poles": [(w - e0).cpu().numpy()] * len(G)}
    h1, l1 = _sector(c, 1)
    times1, look1 = _matrix(H, h1, l1), _Lookup(h1, l1)
    if kind == "ground":
        X, E = _plain_lowest(_matrix(H, hi, lo), n, 1, dev)
        Y = torch.cat([_push(_dipole(nf, k), hi, lo, look1, X, len(h1)) for k in ("Tx", "Tz")], dim=1)
        a, b = _plain_lanczos(times1, Y, NTRI, eps, GAMMA)
        w = _grid(-20.0, 20.0, c["ne"], dev)[None, :] + E.repeat(2)[:, None]
        return {"E": E.cpu().numpy(), "G": _fraction(a, b, w, GAMMA).cpu().numpy()}
    # RIXS
    o = _rixs_options(c)
    x = _vectors(n, 1, seed, True)
    times = _matrix(H, hi, lo)
    e0 = float(_expect(times, x)[0])
    v = _push(_dipole(nf, "Tz"), hi, lo, look1, x, len(h1))
    K, a, b = _plain_krylov(times1, v, NTRI, eps)
    T = torch.diag(a[1:]) + torch.diag(b[1:], 1) + torch.diag(b[1:], -1)
    ev, Z = torch.linalg.eigh(T)
    w1 = _grid(o["Emin1"], o["Emax1"], o["NE1"], dev) + e0
    C = b[0] * torch.einsum("ik,k,pk->ip", Z.to(torch.complex128), Z[0].to(torch.complex128),
                            1 / (w1[:, None] - ev[None, :] + 0.5j * o["Gamma1"]))
    look = _Lookup(hi, lo)
    Y = torch.cat([_push(_dipole(nf, k).dagger(), h1, l1, look, K @ C, n) for k in ("Tx", "Ty", "Tz")], dim=1)
    a2, b2 = _plain_lanczos(times, Y, NTRI, eps, float(np.sqrt(np.finfo(float).eps)) + o["Gamma2"])
    w2 = (_grid(o["Emin2"], o["Emax2"], o["NE2"], dev) + e0)[None, :].expand(Y.shape[1], -1)
    return _fraction(a2, b2, w2, o["Gamma2"]).cpu().numpy()


def _plain_krylov(times, v, ntri, eps):
    """Fully reorthogonalised Lanczos: the vectors as columns, a (ntri + 1), b (ntri)."""
    a = torch.zeros(ntri + 1, dtype=torch.float64, device=v.device)
    b = torch.zeros(ntri, dtype=torch.float64, device=v.device)
    K = torch.zeros((len(v), ntri), dtype=torch.complex128, device=v.device)
    err, w = 1.0, v[:, 0]
    for i in range(ntri):
        if i:
            w = times(K[:, i - 1:i])[:, 0]
            a[i] = torch.vdot(K[:, i - 1], w).real
            for _ in range(2):
                w = w - K[:, :i] @ (K[:, :i].conj().T @ w)
        b[i] = torch.linalg.vector_norm(w)
        w = w / b[i]
        K[:, i] = torch.where(w.abs() > eps / err, w, torch.zeros_like(w))
    w = times(K[:, -1:])[:, 0]
    a[ntri] = torch.vdot(K[:, -1], w).real
    return K, a, b


def _plain_lowest(times, n, k, dev):
    """The lowest k eigenpairs: a fully reorthogonalised Lanczos, long enough to converge."""
    m = min(n, 900)
    g = torch.Generator(device=dev)
    g.manual_seed(1)
    Q = torch.zeros((m, n), dtype=torch.float64, device=dev)
    a = torch.zeros(m, dtype=torch.float64, device=dev)
    b = torch.zeros(m, dtype=torch.float64, device=dev)
    w = torch.randn(n, dtype=torch.float64, device=dev, generator=g)
    for i in range(m):
        if i:
            b[i] = torch.linalg.vector_norm(w)
        Q[i] = w / torch.linalg.vector_norm(w)
        w = times(Q[i][:, None].to(torch.complex128))[:, 0].real
        a[i] = Q[i] @ w
        for _ in range(2):
            w = w - Q[:i + 1].T @ (Q[:i + 1] @ w)
    ev, Z = torch.linalg.eigh(torch.diag(a) + torch.diag(b[1:], 1) + torch.diag(b[1:], -1))
    return (Q.T @ Z[:, :k]).to(torch.complex128), ev[:k]


def _exact_spectra(c, seed):
    """The ligand-field ion: the resolvent itself, by diagonalising H on the determinants it reaches
    (200 steps exhaust that space)."""
    ops, R = workloads.ligand_field()
    H = ops["HX"]
    dets = api.enumerate_restricted(26, R)
    hi, lo = _pairs_of(dets, 26)
    rng = np.random.default_rng(int(seed))
    cols = []
    for _ in range(c["states"]):
        v = rng.standard_normal(len(dets)) * 10.0 ** (-3.0 * rng.random(len(dets)))
        cols.append(v / np.linalg.norm(v))
    X = torch.from_numpy(np.stack(cols, axis=1)).to(hi.device).to(torch.complex128)
    Ts = [ops[k] for k in ("Tx", "Ty", "Tz")[:c["operators"]]]
    grown = [_grown(T, hi, lo) for T in Ts]
    sh, sl = torch.cat([g[0] for g in grown]), torch.cat([g[1] for g in grown])
    while True:
        both = torch.unique(torch.stack([sh, sl], dim=1), dim=0)
        gh, gl = _grown(H, both[:, 0].contiguous(), both[:, 1].contiguous())
        more = torch.unique(torch.cat([both, torch.stack([gh, gl], dim=1)]), dim=0)
        sh, sl = more[:, 0].contiguous(), more[:, 1].contiguous()
        if len(more) == len(both):
            break
    n = len(sh)
    look = _Lookup(sh, sl)
    M = _push(H, sh, sl, look, torch.eye(n, dtype=torch.complex128, device=hi.device), n)
    w, V = torch.linalg.eigh((M + M.conj().T) / 2)
    # <psi|H|psi> on the states' own determinants
    e0 = (X.conj() * _push(H, hi, lo, _Lookup(hi, lo), X, len(hi))).sum(0).real
    G = []
    for T in Ts:
        wt = (V.conj().T @ _push(T, hi, lo, look, X, n)).abs() ** 2
        for j in range(c["states"]):
            om = _grid(-10.0, 20.0, c["ne"], hi.device) + e0[j] + 0.5j * GAMMA
            G.append((wt[None, :, j] / (om[:, None] - w[None, :])).sum(1))
    return torch.stack(G).cpu().numpy()
