"""Performance cases of the line-intensity engine: the work a user's program has it do.

Every case goes through the public Python mirror of the C ABI (``Engine``):

* ``half_ls``   half line strength of one eigenvector (``Engine.half_ls``), host vector in, host result out;
* ``noalloc``   the same on device buffers that the caller owns (``gi_half_ls_noalloc``);
* ``job``       a line-intensity job over consecutive J values (``Engine.run``), its lines sorted as the
                reference prints them and read back into the program's own buffer (the intensity threshold keeps the
                strongest tenth or so of them); ``shards`` > 1: one batch of its initial levels;
* ``serve``     pair jobs submitted to the serving loop, waited for and read back.

Sizes are those of the repository's workloads (triatomic C2v with 200, 2000 and 5000 vibrational functions,
tetratomic C3v with 3000, J up to 40) and ragged ones between them.  Inputs follow the workloads'
distributions: dipole entries N(0,1) exp(-|i-j|/10) or magnitudes log-uniform in 1e-8..1, unit Gaussian
eigenvectors (device resident, as an eigensolver leaves them), sorted uniform energies.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from __graft_entry__ import load_package

GI = load_package()

DEGEN = {"c2v": (1, 1, 1, 1), "c3v": (1, 1, 2)}
PAIRS = {"c2v": (1, 1, 2, 2), "c3v": (1, 1, 2)}
PARTNER = {"c2v": (1, 0, 3, 2), "c3v": (1, 0, 2)}
GNS = {"c2v": (1.0, 1.0, 3.0, 3.0), "c3v": (2.0, 2.0, 2.0)}
SYM = {"c2v": 1, "c3v": 2}


def _case(name, kind, group, N, J, **kw):
    c = {"name": name, "kind": kind, "group": group, "N": N, "J": J, "nj": 1, "nvec": 0, "precision": "split",
         "dipole": "decay", "vib": N, "shards": 1, "gamma": 0, "ideg": 0, "dj": 1, "graph": False,
         "compact": False, "panel": 0, "thresh": 1e-30, "jobs": 0}
    c.update(kw)
    return c


def listed():
    return [
        # one vector of the smallest workload: latency and launches are all there is
        _case("half_ls_small", "half_ls", "c2v", 200, 1, precision="fp64"),
        # an eigensolver's vector against the 2000-function dipole, split precision and FP64
        _case("half_ls_plain", "half_ls", "c2v", 2000, 10, gamma=1),
        _case("half_ls_fp64", "half_ls", "c2v", 2000, 10, gamma=2, dj=0, precision="fp64"),
        # the second degenerate component of an E vector of the tetratomic workload
        _case("half_ls_E", "half_ls", "c3v", 3000, 20, gamma=2, ideg=1, dj=-1),
        # a caller that cannot allocate: device vector to device result, ragged N
        _case("noalloc_ragged", "noalloc", "c2v", 777, 5, gamma=3),
        # the whole smallest workload (J = 0..2, every eigenvector), FP64
        _case("job_small_fp64", "job", "c2v", 200, 0, nj=3, nvec=600, precision="fp64", thresh=1e-19),
        # a reference run (J, J+1) in FP64 at a ragged size
        _case("job_pair_fp64", "job", "c2v", 1013, 3, nj=2, nvec=150, precision="fp64", thresh=1e-21),
        # a batch of the throughput workload as a production loop runs it: split precision, graph replay
        _case("job_plain", "job", "c2v", 2000, 2, nj=5, nvec=1000, shards=16, graph=True, thresh=1e-22),
        # low-J blocks of the tetratomic workload, compact line records
        _case("job_low_j", "job", "c3v", 1500, 0, nj=5, nvec=300, compact=True, thresh=1e-21),
        # a batch of the tetratomic workload at J = 20, 21
        _case("job_batched", "job", "c3v", 3000, 20, nj=2, nvec=1500, shards=12, graph=True, thresh=5e-24),
        # a batch of the precision workload: J = 20, 21, dipole magnitudes over eight decades
        _case("job_precision", "job", "c2v", 5000, 20, nj=2, nvec=2000, vib=2500, dipole="loguniform", shards=32,
              thresh=1e-22),
        # pair jobs arriving at a serving loop (three slots), each block's half line strength computed anew
        _case("serve_pairs", "serve", "c3v", 1200, 4, nj=3, nvec=400, jobs=12, thresh=1e-22),
    ]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["half_ls", "half_ls", "noalloc", "job", "job", "job", "serve"])
    group = rng.choice(["c2v", "c3v"])
    kw = {"precision": rng.choice(["split", "split", "fp64"]), "gamma": rng.randrange(len(DEGEN[group])),
          "dipole": rng.choice(["decay", "decay", "loguniform"])}
    if kind in ("half_ls", "noalloc"):
        N, J = logint(150, 3000 if kind == "half_ls" else 1000), rng.randint(1, 20 if kind == "half_ls" else 6)
        kw["ideg"] = rng.randrange(DEGEN[group][kw["gamma"]])
        kw["dj"] = rng.choice([-1, 0, 1])
        if kind == "noalloc":
            kw["precision"] = "fp64"
        return {k: v for k, v in _case("", kind, group, N, J, **kw).items() if k != "name"}
    fp64 = kw["precision"] == "fp64"
    N = logint(150, 600 if fp64 else 2500)
    J = rng.randint(0, 4 if fp64 else 12)
    nj = rng.randint(2, 3)
    kw.update(nj=nj, nvec=logint(40, 150 if fp64 else 600), thresh=10.0 ** rng.uniform(-24.0, -21.0))
    if kind == "serve":
        kw.update(jobs=rng.randint(3, 10), nvec=min(kw["nvec"], 300), nj=3)
    else:
        kw.update(shards=rng.choice([1, 4, 16]) if not fp64 else rng.choice([1, 4]), graph=rng.random() < 0.4,
                  compact=rng.random() < 0.3)
        if not kw["graph"] and rng.random() < 0.25:
            kw["panel"] = logint(100, max(101, N))
    return {k: v for k, v in _case("", kind, group, N, J, **kw).items() if k != "name"}


# ---------------------------------------------------------------- inputs
def _vib(case, rng):
    """Vibrational functions: C2v irreps (A1 or B2), or C3v levels (A1, A2, or E pairs) as in a contracted basis."""
    N = case["N"]
    if case["group"] == "c2v":
        return np.where(rng.random(N) < 0.5, 0, 3)
    kinds = []
    while len(kinds) < N:
        x = rng.random()
        if x < 0.5 and len(kinds) + 2 <= N:
            kinds += [2, 2]
        else:
            kinds.append(0 if x < 0.8 else 1)
    return np.array(kinds)


class _Basis:
    pass


def _finish(J, nrep, icase, lam, iroot, k, tau, Nsym, mat, rep):
    b = _Basis()
    b.jval, b.Maxcontracts, b.Maxsymcoeffs = J, len(icase), Nsym.shape[0]
    b.max_deg_size = b.mat_size = mat
    b.icontr2icase = np.concatenate([icase, lam]).astype(np.int32)
    b.iroot_correlat_j0, b.k = iroot.astype(np.int32), k.astype(np.int32)
    b.ktau = (2 * k + tau).astype(np.int32)
    b.Nsym = np.ascontiguousarray(Nsym.astype(np.int32)).reshape(-1)
    b.Ntotal = Nsym.sum(axis=0).astype(np.int32)
    b.repres = rep
    return b


def _c2v_basis(J, vib, rng):
    N = len(vib)
    kk = np.concatenate([np.zeros(N, int)] + [np.full(2 * N, k) for k in range(1, J + 1)])
    v = np.concatenate([np.arange(N)] + [np.repeat(np.arange(N), 2)] * J)
    lam = np.concatenate([np.zeros(N, int)] + [np.tile([0, 1], N)] * J)
    tau = np.where(kk == 0, J % 2, lam)
    icase = kk * N + v
    g = vib[v] ^ (((kk & 1) << 1) | ((tau ^ kk) & 1))
    Nsym = np.zeros(((J + 1) * N, 4), int)
    np.add.at(Nsym, (icase, g), 1)
    mat = 1 if J == 0 else 2
    val = rng.choice([-1.0, 1.0], size=len(v))
    rep = []
    for q in range(4):
        roots = np.nonzero(g == q)[0]
        r = np.zeros((mat, max(len(roots), 1)))
        r[lam[roots], np.arange(len(roots))] = val[roots]
        rep.append(r.reshape(-1))
    return _finish(J, 4, icase, lam, v, kk, tau, Nsym, mat, rep)


def _c3v_basis(J, kinds, rng):
    first = [i for i in range(len(kinds)) if kinds[i] != 2]
    e = np.nonzero(kinds == 2)[0][::2]
    start = np.sort(np.concatenate([np.array(first, int), e]))
    kind, nlev = kinds[start], len(start)
    nvi = np.where(kind == 2, 2, 1)
    irr = {(0, 0): [0], (0, 1): [1], (0, 2): [2], (1, 0): [1], (1, 1): [0], (1, 2): [2], (3, 0): [0, 1],
           (3, 1): [0, 1], (3, 2): [2, 2], (2, 0): [2], (2, 1): [2], (2, 2): [0, 1, 2]}
    rot = [J % 2] + [3 if k % 3 == 0 else 2 for k in range(1, J + 1)]
    Nsym = np.zeros((J + 1, nlev, 3), int)
    for k in range(J + 1):
        for q in range(3):
            sel = kind == q
            for x in irr[(rot[k], q)]:
                Nsym[k, sel, x] += 1
    Nsym = Nsym.reshape(-1, 3)
    ij = np.cumsum(Nsym, axis=0) - Nsym
    nl = (np.where(np.arange(J + 1) == 0, 1, 2)[:, None] * nvi[None, :]).reshape(-1)
    icase = np.repeat(np.arange(len(nl)), nl)
    r0 = np.cumsum(nl) - nl
    lam = np.arange(len(icase)) - r0[icase]
    kk, lev = icase // nlev, icase % nlev
    tau = np.where(kk == 0, J % 2, lam // nvi[lev])
    v = start[lev] + lam % nvi[lev]
    tot = Nsym.sum(axis=0)
    mat = int(nl.max())
    rep = [np.zeros((mat, DEGEN["c3v"][g], max(int(tot[g]), 1))) for g in range(3)]
    for k in range(J + 1):
        for q in range(3):
            cases = k * nlev + np.nonzero(kind == q)[0]
            if not len(cases):
                continue
            n = int(nl[cases[0]])
            Q = np.linalg.qr(rng.standard_normal((len(cases), n, n)))[0]
            row = 0
            for g in range(3):
                for j in range(int(Nsym[cases[0], g])):
                    for d in range(DEGEN["c3v"][g]):
                        for il in range(n):
                            rep[g][il, d, ij[cases, g] + j] = Q[:, row, il]
                        row += 1
    return _finish(J, 3, icase, lam, v, kk, tau, Nsym, mat, [r.reshape(-1) for r in rep])


def _dipole(case, seed):
    """[3][f][v]: x and z symmetric, y antisymmetric (drawn on the GPU, handed over in host memory)."""
    N = case["N"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    mu = torch.empty(3, N, N, dtype=torch.float64, device="cuda")
    i = torch.arange(N, device="cuda", dtype=torch.float64)
    for c in range(3):
        if case["dipole"] == "decay":
            a = torch.randn(N, N, generator=gen, dtype=torch.float64, device="cuda")
            a *= torch.exp(-(i[:, None] - i[None, :]).abs() / 10.0)
        else:
            a = 10.0 ** (torch.rand(N, N, generator=gen, dtype=torch.float64, device="cuda") * 8.0 - 8.0)
            a *= torch.where(torch.rand(N, N, generator=gen, device="cuda") < 0.5, -1.0, 1.0)
        u = torch.triu(a, 1)
        mu[c] = u.T - u if c == 1 else torch.triu(a) + u.T
    return mu.cpu().numpy()


class _Params:
    """The INTENSITY block of a deck."""
    ZPE, reduced, thresh_linestrength = 0.0, False, 0.0

    def __init__(self, case, q):
        c2v = case["group"] == "c2v"
        self.temperature, self.q_stat = 296.0 if c2v else 500.0, q
        self.gns, self.isym_pairs, self.nmodes = GNS[case["group"]], PAIRS[case["group"]], 3 if c2v else 6
        self.erange_lower = (0.0, 20000.0 if c2v else 12000.0)
        self.erange_upper = (0.0, 20000.0 if c2v else 16000.0)
        self.freq_window = (0.0, 25000.0 if c2v else 20000.0)
        self.thresh_intensity = case["thresh"]

    def windows(self):
        w = np.array([[0] * self.nmodes, [1 << 30] * self.nmodes], np.int32)
        return w, w


def _model(case, seed):
    """Bases, blocks (device vectors, host energies and quanta) and parameters of a case."""
    rng = np.random.default_rng([seed, 11])
    vib = _vib(case, rng)
    make = _c2v_basis if case["group"] == "c2v" else _c3v_basis
    bases = {}
    vectors = case["kind"] in ("half_ls", "noalloc")
    js = sorted({case["J"], max(0, case["J"] + case["dj"])}) if vectors else range(case["J"], case["J"] + case["nj"])
    for J in js:
        low = vib if J == 0 else vib[:case["vib"]].copy()
        if case["group"] == "c3v" and (low == 2).sum() % 2:
            low[-1] = 0  # an E pair cut at the end
        bases[J] = make(J, low, rng)
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    blocks = {}
    emax, ecut = (20000.0, 15000.0) if case["group"] == "c2v" else (16000.0, 12000.0)
    for J, b in bases.items():
        for g in range(len(DEGEN[case["group"]])):
            n = int(b.Ntotal[g])
            if vectors and (J, g) != (case["J"], case["gamma"]):
                continue
            e = np.sort(rng.uniform(0.0, emax, n))
            e = e[:1] if vectors else e[e < ecut][:case["nvec"]]
            v = torch.randn(len(e), n, generator=gen, dtype=torch.float64, device="cuda")
            v /= v.norm(dim=1, keepdim=True)
            q = np.zeros((len(e), 4 if case["group"] == "c2v" else 7), np.int32)
            q[:, 0] = rng.integers(0, 2 * J + 1, len(e))
            q[:, 1:] = rng.integers(0, 8, q[:, 1:].shape)
            blocks[(J, g)] = (v, e, q)
    T = 296.0 if case["group"] == "c2v" else 500.0
    beta = _PLANCK * _VELLGT / (_BOLTZ * T)
    z = sum(GNS[case["group"]][g] * (2 * J + 1) * np.exp(-e * beta).sum() for (J, g), (_, e, _q) in blocks.items())
    return bases, blocks, _Params(case, float(z) or 1.0)


def _serve_list(case, blocks):
    """The pair jobs of a serving case, in arrival order (block pairs that can carry lines)."""
    jobs = []
    for (J, g), (v, _, _) in sorted(blocks.items()):
        for jF in (J - 1, J, J + 1):
            f = blocks.get((jF, PARTNER[case["group"]][g]))
            if len(v) and f is not None and len(f[0]) and J + jF >= 1 and not J == jF == case["J"]:
                jobs.append((J, g, jF, PARTNER[case["group"]][g]))
    order = np.random.default_rng(5).permutation(len(jobs))
    return [jobs[i] for i in order[:case["jobs"]]]


def prepare(case, seed):
    bases, blocks, params = _model(case, seed)
    mu = _dipole(case, seed)
    eng = GI.Engine(0)
    eng.set_symmetry(SYM[case["group"]])
    eng.set_params(params, precision=GI.GI_PREC_SPLIT if case["precision"] == "split" else GI.GI_PREC_FP64)
    if case["panel"]:
        eng.set_dipole_streamed(case["N"], mu, case["panel"])
    else:
        eng.set_dipole(case["N"], mu)
    for J in sorted(bases):
        eng.set_basis(bases[J])
    state = {"case": case, "eng": eng}
    if case["kind"] in ("half_ls", "noalloc"):
        jF = max(0, case["J"] + case["dj"])
        v = blocks[(case["J"], case["gamma"])][0][0].contiguous()
        state["call"] = (case["J"], case["gamma"], case["ideg"], jF)
        state["D"] = bases[jF].Maxcontracts
        if case["kind"] == "half_ls":
            state["v"] = v.cpu().numpy()
        else:
            state["v"], state["out"] = v, torch.empty(state["D"], dtype=torch.float64, device="cuda")
        return state
    for (J, g), (v, e, q) in sorted(blocks.items()):
        torch.cuda.synchronize()
        eng.set_block_device(J, g, v.data_ptr(), v.shape[0], v.shape[1], e, q)
    state["lines"] = np.zeros(_cap(case), GI.LINE_COMPACT_DTYPE if case["compact"] else GI.LINE_DTYPE)
    if case["kind"] == "serve":
        state["jobs"] = _serve_list(case, blocks)
        state["lines"] = np.zeros((len(state["jobs"]), _cap(case)), GI.LINE_DTYPE)
        eng.serve_start(slots=3, budget=16 << 30, zcache=False)
    return state


# ---------------------------------------------------------------- one pass
def _cap(case):
    """Lines a buffer holds: emission and absorption pairs of all blocks, a little over half of them absorption
    (a serving case: of one pair job)."""
    n = case["nvec"]
    if case["kind"] == "serve":
        return n * n
    return 1000 + int(0.6 * n * n / case["shards"] * len(DEGEN[case["group"]]) * (3 * case["nj"] - 3))


def _columns(lines):
    names = [f for f in ("level_i", "level_f", "nu", "S", "A", "I", "t") if f in lines.dtype.names]
    return {f: lines[f] for f in names}


def run(state):
    case, eng = state["case"], state["eng"]
    if case["kind"] == "half_ls":
        return eng.half_ls(*state["call"], state["v"], state["D"])
    if case["kind"] == "noalloc":
        jI, g, d, jF = state["call"]
        st = GI.lib().gi_half_ls_noalloc(eng._h, jI, g, d, jF, ctypes.c_void_p(state["v"].data_ptr()),
                                         ctypes.c_void_p(state["out"].data_ptr()),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != GI.GI_OK:
            raise GI.GiError(st, "gi_half_ls_noalloc")
        return state["out"]
    buf = state["lines"]
    if case["kind"] == "job":
        n = eng.run(graph=case["graph"], compact=case["compact"], nshards=case["shards"])
        if n > len(buf):
            raise RuntimeError("%d lines, room for %d" % (n, len(buf)))
        eng.sort_lines()
        get = GI.lib().gi_get_lines_compact if case["compact"] else GI.lib().gi_get_lines
        if n and get(eng._h, 0, n, buf.ctypes.data) != GI.GI_OK:
            raise RuntimeError("reading the lines")
        return {"n": n, **_columns(buf)}
    count = np.zeros(len(state["jobs"]), np.int64)
    for k, i in enumerate([eng.submit(*j) for j in state["jobs"]]):
        lines = eng.job_lines(i)
        count[k] = len(lines)
        buf[k, :len(lines)] = lines[np.lexsort((lines["level_f"], lines["level_i"]))]
    return {"n": count, **_columns(buf)}


# ---------------------------------------------------------------- the work of a pass
def work(case):
    """FP64 operations and bytes the path cannot do without: only products that the selection rules leave."""
    c2v = case["group"] == "c2v"
    N, vib, ng = case["N"], case["vib"], 4 if c2v else 3
    share_k, share = (0.5, 0.25) if c2v else (0.78, 0.66)  # of v alone; of (v, f) pairs
    if case["kind"] in ("half_ls", "noalloc"):
        nslot, jF = 2 * case["J"] + 1, max(0, case["J"] + case["dj"])
        io = 8.0 * (nslot * vib / 3 + (2 * jF + 1) * vib)
        return {"bytes": 8.0 * 3 * vib * vib + io, "flops": 2.0 * 3 * vib * vib * nslot * share_k}
    fl = by = 0.0
    js = range(case["J"], case["J"] + case["nj"])

    def nvec(J):
        return min(case["nvec"], int((2 * J + 1) * vib / 4 * 0.75))

    npair = 0
    for J in js:
        nI = nvec(J) / case["shards"]
        for jF in js:
            if abs(J - jF) <= 1 and J + jF >= 1 and not J == jF == case["J"]:
                npair += ng
                fl += ng * 2.0 * (2 * jF + 1) * vib / 4 * nI * nvec(jF) * (1 if c2v else 2)
        fl += ng * nI * (1 if c2v else 4 / 3) * (2 * J + 1) * 2.0 * 3 * vib * vib * share
        by += ng * 8.0 * nvec(J) * (2 * J + 1) * vib / 4
    if case["kind"] == "serve":
        fl *= min(1.0, case["jobs"] / max(1, npair))
    return {"bytes": by + 8.0 * 3 * vib * vib, "flops": fl}


# ---------------------------------------------------------------- the same in plain 64 bits
_PLANCK, _VELLGT, _BOLTZ, _AVOGNO = 6.62606896e-27, 2.99792458e10, 1.380658e-16, 6.0221415e23


@functools.lru_cache(maxsize=None)
def _threej(a, b, c, al, be, ga):
    """Wigner 3j by Racah's sum over exact integers."""
    f = math.factorial
    if al + be + ga or c > a + b or c < abs(a - b) or abs(al) > a or abs(be) > b or abs(ga) > c:
        return 0.0
    s = 0.0
    pre = math.sqrt(f(a + b - c) * f(a - b + c) * f(b + c - a) / f(a + b + c + 1)) * math.sqrt(
        float(f(a + al) * f(a - al)) * float(f(b + be) * f(b - be))) * math.sqrt(float(f(c + ga) * f(c - ga)))
    for t in range(max(0, b - c - al, a + be - c), min(a + b - c, a - al, b + be) + 1):
        d = f(t) * f(c - b + t + al) * f(c - a + t - be) * f(a + b - c - t) * f(a - t - al) * f(b - t + be)
        s += (-1) ** t / d
    return (-1) ** (a - b - ga) * pre * s


def _terms(jI, jF):
    """(kF, tauF) -> [(kI, tauI, component, coefficient)] of the half line strength."""
    out = {}
    for kF in range(jF + 1):
        for tF in (0, 1):
            for kI in range(max(kF - 1, 0), min(kF + 1, jI) + 1):
                for tI in (0, 1):
                    c, L = (2, tF - tI) if kF == kI else (0, (tF - tI) * (kF - kI)) if tF != tI else (1, -1)
                    sign = (-1) ** ((kF % 3) * tF + (kI % 3) * tI + kI)
                    x = sign * L * _threej(jI, 1, jF, kI, kF - kI, -kF)
                    x *= 1 / math.sqrt(2.0) if kI != kF and kI * kF else 1.0
                    if x:
                        out.setdefault((kF, tF), []).append((kI, tI, c, x))
    return out


def _primitive(b, g, ndeg, d, vecs):
    """Symmetrised vectors [n][nsize] in the primitive basis [n][D], component d."""
    dev, D = vecs.device, b.Maxcontracts
    case, lam = b.icontr2icase[:D], b.icontr2icase[D:]
    nsym = b.Nsym.reshape(b.Maxsymcoeffs, -1)[:, g]
    it = np.cumsum(nsym) - nsym
    nt = max(int(b.Ntotal[g]), 1)
    rep = b.repres[g].reshape(b.mat_size, ndeg, nt)
    out = torch.zeros(vecs.shape[0], D, dtype=torch.float64, device=dev)
    for j in range(int(nsym.max(initial=0))):
        r = np.nonzero(nsym[case] > j)[0]
        s = it[case[r]] + j
        out[:, torch.from_numpy(r).to(dev)] += vecs[:, torch.from_numpy(s).to(dev)] * torch.from_numpy(
            rep[lam[r], d, s]).to(dev)
    return out


def _half(bI, bF, prim, mu):
    """Half line strength [n][D_F] of primitive initial vectors [n][D_I]."""
    dev, N = prim.device, mu.shape[1]
    n, ktI = prim.shape[0], bI.ktau
    out = torch.zeros(n, bF.Maxcontracts, dtype=torch.float64, device=dev)
    y = {}
    for key in np.unique(ktI):
        r = np.nonzero(ktI == key)[0]
        y[int(key)] = torch.zeros(n, N, dtype=torch.float64, device=dev)
        y[int(key)][:, torch.from_numpy(bI.iroot_correlat_j0[r].astype(np.int64)).to(dev)] = prim[
            :, torch.from_numpy(r).to(dev)]
    z = {}
    for (kF, tF), terms in _terms(bI.jval, bF.jval).items():
        r = np.nonzero(bF.ktau == 2 * kF + tF)[0]
        if not len(r):
            continue
        acc = 0.0
        for kI, tI, c, x in terms:
            key = 2 * kI + tI
            if key in y:
                if (key, c) not in z:
                    z[(key, c)] = y[key] @ mu[c].T
                acc = acc + x * z[(key, c)]
        if torch.is_tensor(acc):
            v = torch.from_numpy(bF.iroot_correlat_j0[r].astype(np.int64)).to(dev)
            out[:, torch.from_numpy(r).to(dev)] = acc[:, v]
    return out


def _project(b, g, ndeg, d, h):
    """Primitive half line strength [n][D] on the symmetrised basis [n][nsize], component d."""
    dev, D = h.device, b.Maxcontracts
    case, lam = b.icontr2icase[:D], b.icontr2icase[D:]
    nsym = b.Nsym.reshape(b.Maxsymcoeffs, -1)[:, g]
    it = np.cumsum(nsym) - nsym
    nt = max(int(b.Ntotal[g]), 1)
    rep = b.repres[g].reshape(b.mat_size, ndeg, nt)
    out = torch.zeros(h.shape[0], int(b.Ntotal[g]), dtype=torch.float64, device=dev)
    for j in range(int(nsym.max(initial=0))):
        r = np.nonzero(nsym[case] > j)[0]
        s = it[case[r]] + j
        out.index_add_(1, torch.from_numpy(s).to(dev), h[:, torch.from_numpy(r).to(dev)] * torch.from_numpy(
            rep[lam[r], d, s]).to(dev))
    return out


def exact(case, seed):
    bases, blocks, P = _model(case, seed)
    mu = torch.from_numpy(_dipole(case, seed)).to("cuda")
    deg = DEGEN[case["group"]]
    if case["kind"] in ("half_ls", "noalloc"):
        J, g, jF = case["J"], case["gamma"], max(0, case["J"] + case["dj"])
        v = blocks[(J, g)][0]
        h = _half(bases[J], bases[jF], _primitive(bases[J], g, deg[g], case["ideg"], v), mu)[0]
        return h.cpu().numpy() if case["kind"] == "half_ls" else h
    lv = [(float(x), J, g, r) for J in sorted(bases) for g in range(len(deg)) for r, x in enumerate(blocks[(J, g)][1])
          if 0.0 <= x <= max(P.erange_lower[1], P.erange_upper[1])]
    lv.sort(key=lambda x: x[0])
    ids = {k: np.full(len(b[1]), -1, np.int64) for k, b in blocks.items()}
    for n, (_, J, g, r) in enumerate(lv):
        ids[(J, g)][r] = n
    beta = _PLANCK * _VELLGT / (_BOLTZ * P.temperature)
    A0 = 64.0e-36 * math.pi ** 4 / (3.0 * _PLANCK)
    I0 = 8.0e-36 * math.pi ** 3 * _AVOGNO / (3.0 * _PLANCK * _VELLGT)

    def pair(J, g, jF, gF, recs):
        (vI, eI, _), (vF, eF, _) = blocks[(J, g)], blocks[(jF, gF)]
        T = torch.zeros(len(recs), len(eF), 4, dtype=torch.float64, device="cuda")
        for d in range(deg[g]):
            h = _half(bases[J], bases[jF], _primitive(bases[J], g, deg[g], d, vI[torch.from_numpy(recs).cuda()]), mu)
            for dF in range(deg[gF]):
                T[:, :, d + 2 * dF] = _project(bases[jF], gF, deg[gF], dF, h) @ vF.T
        T = T.cpu().numpy()
        nu = eF[None, :] - eI[recs][:, None]
        ls = (T * T).sum(axis=2) / deg[g]
        S = ls * P.gns[g] * ((2 * J + 1) * (2 * jF + 1))
        I = S * I0 * np.abs(nu) * np.exp(-eI[recs] * beta)[:, None] * (1.0 - np.exp(-np.abs(nu) * beta)) / P.q_stat
        A = A0 * (2 * J + 1) * ls * np.abs(nu) ** 3
        ok = (nu >= P.freq_window[0]) & (nu <= P.freq_window[1]) & (I / _AVOGNO >= P.thresh_intensity)
        ok &= (eF >= P.erange_upper[0])[None, :] & (eF <= P.erange_upper[1])[None, :]
        i, f = np.nonzero(ok)
        return i, f, {"nu": nu[i, f], "S": S[i, f], "A": A[i, f], "I": I[i, f], "t": T[i, f]}

    def lower(J, g):
        e = blocks[(J, g)][1]
        return np.nonzero((e >= P.erange_lower[0]) & (e <= P.erange_lower[1]))[0]

    if case["kind"] == "serve":
        jobs = _serve_list(case, blocks)
        out = np.zeros((len(jobs), _cap(case)), GI.LINE_DTYPE)
        count = np.zeros(len(jobs), np.int64)
        for k, (J, g, jF, gF) in enumerate(jobs):
            recs = lower(J, g)
            i, f, col = pair(J, g, jF, gF, recs)
            count[k] = len(i)
            for name, x in {"level_i": recs[i], "level_f": f, **col}.items():
                out[name][k, :len(i)] = x
        return {"n": count, **_columns(out)}
    parts = []
    for (J, g) in sorted(blocks):
        recs = lower(J, g)
        recs = recs[ids[(J, g)][recs] % case["shards"] == 0]
        gF = PARTNER[case["group"]][g]
        for jF in (J - 1, J, J + 1):
            if jF in bases and J + jF >= 1 and not J == jF == case["J"] and len(recs) and len(blocks[(jF, gF)][1]):
                i, f, col = pair(J, g, jF, gF, recs)
                parts.append({"level_i": ids[(J, g)][recs[i]], "level_f": ids[(jF, gF)][f], **col})
    col = {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
    order = np.lexsort((col["level_f"], col["level_i"]))
    out = np.zeros(_cap(case), GI.LINE_COMPACT_DTYPE if case["compact"] else GI.LINE_DTYPE)
    for k in _columns(out):
        out[k][:len(order)] = col[k][order]
    return {"n": len(order), **_columns(out)}
