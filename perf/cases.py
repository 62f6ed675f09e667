"""Performance cases of the two-site hot path, through the entry points a program calls.

A case is one call of ``qcmpodmrg_b200.mpo_dmrg_kernel`` (HVec, HDiag, renorm, pRDM, SVec)
at one dot of a K-orbital chain with bond dimension D, or one half sweep of the driver.
The MPO is the real one (seeded synthetic integrals, decay 3); the bonds carry (N, Sz)
sectors spread as ``qcmpodmrg_b200.synthetic`` spreads them; environments, site tensors and
wavefunctions are random numbers in the blocks that symmetry allows, which is every element
the kernels touch.

kind      what it stands for
hvec      one Davidson product H_eff.psi (the inner loop of every run): FP64 (parity runs),
          f32 and tf32x3 (the mixed-precision runs); device vectors, or host vectors as the
          reference's own Davidson passes them (host=True).  A low-precision product is kept
          in FP32, the precision it has.
hdiag     the Davidson diagonal, once per dot
renorm    the environments of one site after its decimation, once per dot (plans included:
          the site tensor's sectors are new each time); status L or R
prdm      the decimation's density matrix with the noise term, once per dot of a noisy sweep
sp        one product pair (H.c, S.c) of the spin-projected solver
sweep     a half sweep of a small system from a random start state: dots, Davidson,
          decimation and renormalisation together
"""
import numpy
import torch

from qcmpodmrg_b200 import mpo_dmrg_kernel as kern
from qcmpodmrg_b200.dmrg import DMRG, SiteTensor, L_STATUS, R_STATUS, PSI_STATUS
from qcmpodmrg_b200.hamiltonian import make_hamiltonian
from qcmpodmrg_b200.kernels import TensorSet
from qcmpodmrg_b200.mpo import QPHYS, build_mpo
from qcmpodmrg_b200.qtensor import Layout, classification
from qcmpodmrg_b200.spin import SPDMRG, build_mpo_sp, rotation_set, s2quad
from qcmpodmrg_b200.synthetic import random_mps

DECAY = 3.0
NOISE = 1e-4
ENV_STATUS = (True, False, True)


def listed():
    return [
        # the smallest systems of the tests: launches and host work
        {"name": "hvec_K6_D16_f64", "kind": "hvec", "K": 6, "D": 16, "site": 2, "precision": "f64", "host": False},
        # the validation run (K=12, D=100) driven by a host Davidson, vectors copied both ways
        {"name": "hvec_K12_D100_f64_host", "kind": "hvec", "K": 12, "D": 100, "site": 5, "precision": "f64",
         "host": True},
        # an odd bond dimension at a dot near the chain's end, FP32 on the CUDA cores
        {"name": "hvec_K16_D173_f32", "kind": "hvec", "K": 16, "D": 173, "site": 4, "precision": "f32",
         "host": False},
        # mid-chain products of the convergence runs (K=24, D=200)
        {"name": "hvec_K24_D200_tf32x3", "kind": "hvec", "K": 24, "D": 200, "site": 11, "precision": "tf32x3",
         "host": False},
        {"name": "hvec_K24_D200_f64", "kind": "hvec", "K": 24, "D": 200, "site": 11, "precision": "f64",
         "host": False},
        # the benchmark's mid-chain products (K=24, D=500)
        {"name": "hvec_K24_D500_tf32x3", "kind": "hvec", "K": 24, "D": 500, "site": 11, "precision": "tf32x3",
         "host": False},
        {"name": "hvec_K24_D500_f64", "kind": "hvec", "K": 24, "D": 500, "site": 11, "precision": "f64",
         "host": False},
        # once per dot of the benchmark's sweeps: diagonal and environments
        {"name": "hdiag_K24_D300", "kind": "hdiag", "K": 24, "D": 300, "site": 12},
        {"name": "renorm_L_K24_D500", "kind": "renorm", "K": 24, "D": 500, "site": 11, "status": "L"},
        # a noisy warm-up sweep of the validation run
        {"name": "prdm_R_K12_D100", "kind": "prdm", "K": 12, "D": 100, "site": 5, "status": "R"},
        # spin projection at the size the benchmark's sp workload runs
        {"name": "sp_K8_D64", "kind": "sp", "K": 8, "D": 64, "site": 3, "npts": 4},
        # a whole half sweep of a small system
        {"name": "sweep_K8_D32", "kind": "sweep", "K": 8, "D": 32},
    ]


def draw(rng):
    kind = rng.choice(["hvec"] * 6 + ["hdiag", "renorm", "renorm", "prdm", "sp"])
    size = lambda lo, hi: int(round(lo * (hi / float(lo)) ** rng.random()))       # log-uniform
    if kind == "hvec":
        K = rng.randint(6, 24)
        return {"kind": kind, "K": K, "D": size(16, 500), "site": rng.randint(1, K - 3),
                "precision": rng.choice(["f64", "f64", "f32", "tf32x3", "tf32x3"]), "host": rng.random() < 0.2}
    if kind == "hdiag":
        K = rng.randint(6, 24)
        return {"kind": kind, "K": K, "D": size(16, 300), "site": rng.randint(1, K - 3)}
    if kind == "renorm":
        K = rng.randint(6, 24)
        return {"kind": kind, "K": K, "D": size(16, 500), "site": rng.randint(1, K - 3), "status": rng.choice("LR")}
    if kind == "prdm":
        K = rng.randint(6, 14)
        return {"kind": kind, "K": K, "D": size(16, 120), "site": rng.randint(1, K - 3), "status": rng.choice("LR")}
    K = rng.randint(4, 8)
    return {"kind": kind, "K": K, "D": size(12, 64), "site": rng.randint(1, K - 3), "npts": rng.randint(2, 4)}


# ------------------------------------------------------------------ inputs
def _comb(n, k):
    out = 1
    for i in range(k):
        out = out * (n - i) // (i + 1)
    return out


def bond(K, N, sites, D):
    """Quantum numbers of a bond's states, sector by sector: a block of ``sites`` orbitals at
    the left or right end of the chain, up to D states spread over (N, Sz) with Gaussian
    weights around its mean filling (widths of qcmpodmrg_b200.synthetic.random_mps), each
    sector at most as large as the block, and the rest of the chain, can make it."""
    rest = K - sites
    nbar = N * sites / float(K)
    sec = []
    for na in range(sites + 1):
        for nb in range(sites + 1):
            n, s2 = na + nb, na - nb
            ra, rb = N // 2 - na, N // 2 - nb
            if not (0 <= ra <= rest and 0 <= rb <= rest):
                continue
            cap = min(_comb(sites, na) * _comb(sites, nb), _comb(rest, ra) * _comb(rest, rb))
            w = numpy.exp(-0.5 * ((n - nbar) / 0.9) ** 2 - 0.5 * (0.5 * s2 / 0.6) ** 2)
            sec.append((n, 0.5 * s2, cap, w))
    wmax = max(s[3] for s in sec)
    sec = sorted(s for s in sec if s[3] >= 1e-3 * wmax)
    wsum = sum(s[3] for s in sec)
    cnt = [min(s[2], int(numpy.floor(D * s[3] / wsum + 0.5))) for s in sec]
    order = sorted(range(len(sec)), key=lambda i: -sec[i][3])
    while sum(cnt) > D:
        i = max(range(len(sec)), key=lambda j: cnt[j])
        cnt[i] -= 1
    grow = True
    while sum(cnt) < D and grow:
        grow = False
        for i in order:
            if cnt[i] < sec[i][2] and sum(cnt) < D:
                cnt[i] += 1
                grow = True
    q = [[s[0], s[1]] for s, c in zip(sec, cnt) for _ in range(c)]
    return numpy.array(q, dtype=numpy.float64)


def nelec(K):
    return K - K % 2


def _random(n, gen, dev, scale=1.0):
    return torch.randn(n, generator=gen, dtype=torch.float64, device=dev) * scale


class _Dot(DMRG):
    """A DMRG object that holds the MPO of the dot's two sites only."""
    sites = ()

    def _setup_operators(self, ham):
        self.nops = ham.sbas
        self.opers = list(range(ham.sbas))
        self.hpwts = numpy.ones(self.nops)
        self.qkey = numpy.array([float(ham.nelec), self.sz])
        mpo = build_mpo(ham, self.sites)
        self.mpo = {i: TensorSet(l, v, device=self.device) for i, (l, v) in mpo.items()}


class _SPDot(SPDMRG):
    """The same for the spin-projected problem."""
    sites = ()

    def _setup_operators(self, ham):
        self.qpts, self.qwts = s2quad(self.npts, self.sval, self.sz, self.quad)
        self.nops = ham.sbas * self.npts
        self.opers = [x // self.npts for x in range(self.nops)]
        self.hpwts = numpy.array([self.qwts[x % self.npts] for x in range(self.nops)])
        self.qkey = numpy.array([float(ham.nelec), self.sz])
        mpo = build_mpo_sp(ham, self.qpts, self.sites)
        self.mpo = {i: TensorSet(l, v, device=self.device) for i, (l, v) in mpo.items()}
        self.pops = rotation_set(self.qpts, self.device)
        self.popers = [0] * self.npts


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _env(mpo_q, mpo_n, bond_q, nq, gen, dev):
    """Random environments of every operator: index 0 the MPO bond, 1 and 2 the MPS bond in
    its (N, Sz) sectors, with nq quantum numbers (1: N only, under spin projection)."""
    q, n, _ = classification(bond_q)
    lays = [Layout(ENV_STATUS, [mq, q[:, :nq], q[:, :nq]], [mn, n, n]) for mq, mn in zip(mpo_q, mpo_n)]
    return TensorSet(lays, _random(sum(l.size for l in lays), gen, dev, 1.0 / max(1, len(bond_q)) ** 0.5), device=dev)


def _masked(shape_q, status, gen, dev):
    """A random dense tensor that is zero outside the blocks symmetry allows."""
    tot = 0
    for k, (q, s) in enumerate(zip(shape_q, status)):
        v = torch.from_numpy(numpy.rint(2 * numpy.asarray(q))).to(dev)
        v = v.reshape((1,) * k + (len(q),) + (1,) * (len(shape_q) - 1 - k) + (v.shape[-1],))
        tot = tot - v if s else tot + v
    return _random(tuple(len(q) for q in shape_q), gen, dev) * (tot == 0).all(dim=-1)


def _dot(case, seed):
    """The dot's DMRG object with random environments, and the generator for what follows."""
    K, D, i = case["K"], case["D"], case["site"]
    N, sp = nelec(K), case["kind"] == "sp"
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    ham = make_hamiltonian(K, N, 1 + int(seed) % 1000, DECAY)
    if sp:
        cls = type("SPDot", (_SPDot,), {"sites": (i, i + 1)})
        d = cls(ham, case["npts"], device=dev)
    else:
        cls = type("Dot", (_Dot,), {"sites": (i, i + 1)})
        d = cls(ham, device=dev, precision=case.get("precision", "f64"))
    ql, qr = bond(K, N, i, D), bond(K, N, K - i - 2, D)
    d.qnuml, d.qnumr = [None] * (K + 1), [None] * (K + 1)
    d.qnuml[i], d.qnumr[i + 2] = ql, qr
    nq = 1 if sp else 2
    env = lambda lays, k, sign, q: _env([sign * l.qsyms[k] for l in lays], [l.ndims[k] for l in lays],     # noqa: E731
                                        q, nq, gen, dev)
    d.lenv = {i - 1: env(d.mpo[i].layouts, 0, 1.0, ql)}
    d.renv = {i + 2: env(d.mpo[i + 1].layouts, 1, -1.0, qr)}
    if sp:
        d.plenv = {i - 1: env(d.pops.layouts, 0, 1.0, ql)}
        d.prenv = {i + 2: env(d.pops.layouts, 1, -1.0, qr)}
    return d, gen


def _psi_layout(d, i):
    cls = [classification(q) for q in (d.qnuml[i], QPHYS, QPHYS, d.qkey - d.qnumr[i + 2])]
    return Layout(PSI_STATUS, [c[0] for c in cls], [c[1] for c in cls])


def _site_qnums(case, d):
    """Bond quantum numbers of the site tensor a renorm case contracts with."""
    K, N, D, i = case["K"], nelec(case["K"]), case["D"], case["site"]
    if case["status"] == "L":
        return [d.qnuml[i], QPHYS, bond(K, N, i + 1, D)], L_STATUS
    return [bond(K, N, K - i - 1, D), QPHYS, d.qnumr[i + 2]], R_STATUS


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        K, D = case["K"], case["D"]
        d = DMRG(make_hamiltonian(K, nelec(K), 1 + int(seed) % 1000, DECAY), device=_device())
        d.load_mps(random_mps(K, nelec(K), D, int(seed)))
        return {"case": case, "dmrg": d}
    d, gen = _dot(case, seed)
    i = case["site"]
    st = {"case": case, "dmrg": d}
    st["info"] = [d, i, 2, [[d.lenv[i - 1], d.renv[i + 2]]], case.get("status", "L"), True]
    if kind in ("hvec", "hdiag", "sp"):
        lay = _psi_layout(d, i)
        x = _random(lay.size, gen, d.device)
        st["x"] = x.cpu().numpy() if case.get("host") else x
        kern.HDiag(st["info"], lay.size, None)          # compiles the dot's plans, as a solver's first call does
        if kind == "sp":
            kern._sops(d, i)
        st["n"] = lay.size
    elif kind == "renorm":
        q, status = _site_qnums(case, d)
        st["site"] = SiteTensor(_masked(q, status, gen, d.device), q, status, d.device)
    else:
        d.noise = NOISE
        c = _masked([d.qnuml[i], QPHYS, QPHYS, d.qkey - d.qnumr[i + 2]], PSI_STATUS, gen, d.device)
        l, r = c.shape[0], c.shape[3]
        st["x"] = (c / torch.linalg.norm(c)).reshape((1, l, 4, 4 * r) if case["status"] == "L" else (1, 4 * l, 4, r))
    return st


# ------------------------------------------------------------------ one pass
def run(state):
    case, d = state["case"], state["dmrg"]
    kind = case["kind"]
    if kind == "sweep":
        d.psi0 = None
        nmvp, e, dwt, elst, dlst = d.sweep("R", case["D"], 1e-7)
        return {"energies": numpy.array(elst), "kept": numpy.array([len(q) for q in d.qnumr[1:]])}
    if kind == "hvec":
        y = kern.HVec(state["x"], state["info"], state["n"], None)
        if case["precision"] == "f64":
            return y
        return y.astype(numpy.float32) if case["host"] else y.to(torch.float32)
    if kind == "hdiag":
        return kern.HDiag(state["info"], state["n"], None)
    if kind == "sp":
        return [kern.HVec(state["x"], state["info"], state["n"], None),
                kern.SVec(state["x"], state["info"], state["n"], None)]
    if kind == "renorm":
        i, status = case["site"], case["status"]
        kern.renorm(d, i, 2, state["info"][3], None, state["site"], status)
        return d.lenv[i].values if status == "L" else d.renv[i + 1].values
    return kern.pRDM(state["x"], state["info"])


# ------------------------------------------------------------------ the same in 64 bits
_INDEX = {}


def _unpack_index(lay):
    """Row-major position, in the sector-ordered dense tensor, of every packed element: blocks
    allowed by symmetry in row-major order of their sectors, each block row-major."""
    hit = _INDEX.get(id(lay))
    if hit is not None and hit[0] is lay:
        return hit[1]
    off = [numpy.concatenate([[0], numpy.cumsum(n)]) for n in lay.ndims]
    shape = [int(o[-1]) for o in off]
    tot = 0
    for k in range(len(shape)):
        q = numpy.rint(2 * numpy.asarray(lay.qsyms[k]))
        q = q.reshape((1,) * k + (len(q),) + (1,) * (len(shape) - 1 - k) + (q.shape[-1],))
        tot = tot - q if lay.status[k] else tot + q
    parts = []
    for blk in numpy.argwhere((tot == 0).all(axis=-1)):
        lin = numpy.zeros(1, dtype=numpy.int64)
        for k, s in enumerate(blk):
            lin = (lin[:, None] * shape[k] + numpy.arange(off[k][s], off[k][s + 1])[None, :]).ravel()
        parts.append(lin)
    idx = numpy.concatenate(parts) if parts else numpy.zeros(0, dtype=numpy.int64)
    if len(_INDEX) > 64:
        _INDEX.clear()
    _INDEX[id(lay)] = (lay, (shape, idx))
    return shape, idx


def _dense(lay, values):
    shape, idx = _unpack_index(lay)
    out = torch.zeros(int(numpy.prod(shape)), dtype=torch.float64, device=values.device)
    out[torch.from_numpy(idx).to(values.device)] = values
    return out.reshape(shape)


def _packed(lay, dense):
    return dense.reshape(-1)[torch.from_numpy(_unpack_index(lay)[1]).to(dense.device)]


def _sets(tset):
    for lay, off in zip(tset.layouts, tset.offsets):
        yield lay, tset.values[int(off):int(off) + lay.size]


def _chain(psi, L, R, W1, W2, weights):
    out = torch.zeros_like(psi)
    l, r = psi.shape[0], psi.shape[3]
    for w, (ll, lv), (rl, rv), (al, av), (bl, bv) in zip(weights, _sets(L), _sets(R), _sets(W1), _sets(W2)):
        t = _dense(ll, lv)
        t = (t.reshape(-1, l) @ psi.reshape(l, -1)).reshape(t.shape[0], l, 4, 4, r)             # a l n m r
        t = torch.tensordot(_dense(al, av), t, ([0, 3], [0, 2]))                                # b n' l m r
        t = torch.tensordot(_dense(bl, bv), t, ([0, 3], [0, 3]))                                # c m' n' l r
        t = torch.tensordot(t, _dense(rl, rv), ([0, 4], [0, 2]))                                # m' n' l r'
        out += float(w) * t.permute(2, 1, 0, 3)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep" or (not torch.cuda.is_available() and case["D"] > 40):
        return None
    st = prepare(case, seed)
    d, i = st["dmrg"], case["site"]
    L, R, W1, W2 = d.lenv[i - 1], d.renv[i + 2], d.mpo[i], d.mpo[i + 1]
    if kind in ("hvec", "sp"):
        lay = _psi_layout(d, i)
        x = torch.as_tensor(st["x"]).to(d.device)
        psi = _dense(lay, x)
        y = _packed(lay, _chain(psi, L, R, W1, W2, d.hpwts))
        if kind == "hvec":
            return y
        return [y, _packed(lay, _chain(psi, d.plenv[i - 1], d.prenv[i + 2], d.pops, d.pops, d.qwts))]
    if kind == "hdiag":
        lay = _psi_layout(d, i)
        out = 0
        for w, (ll, lv), (rl, rv), (al, av), (bl, bv) in zip(d.hpwts, _sets(L), _sets(R), _sets(W1), _sets(W2)):
            t = torch.diagonal(_dense(ll, lv), dim1=1, dim2=2)                                  # a l
            t = torch.tensordot(t, torch.diagonal(_dense(al, av), dim1=2, dim2=3), ([0], [0]))  # l b n
            t = torch.tensordot(t, torch.diagonal(_dense(bl, bv), dim1=2, dim2=3), ([1], [0]))  # l n c m
            t = torch.tensordot(t, torch.diagonal(_dense(rl, rv), dim1=1, dim2=2), ([2], [0]))  # l n m r
            out = out + float(w) * t
        return _packed(lay, out)
    if kind == "renorm":
        site = st["site"].dense
        left = case["status"] == "L"
        parts = []
        for (el, ev), (wl, wv) in zip(_sets(L if left else R), _sets(W1 if left else W2)):
            e, w = _dense(el, ev), _dense(wl, wv)
            if left:         # out[b, r, r'] = site[l, n', r] E[a, l, l'] W[a, b, n', n] site[l', n, r']
                t = torch.tensordot(e, site, ([2], [0]))                # a l n r'
                t = torch.tensordot(w, t, ([0, 3], [0, 2]))             # b n' l r'
                t = torch.tensordot(t, site, ([1, 2], [1, 0])).permute(0, 2, 1)
            else:            # out[a, l, l'] = site[l, n', r] E[b, r, r'] W[a, b, n', n] site[l', n, r']
                t = torch.tensordot(e, site, ([2], [2]))                # b r l' n
                t = torch.tensordot(w, t, ([1, 3], [0, 3]))             # a n' r l'
                t = torch.tensordot(t, site, ([1, 2], [1, 2])).permute(0, 2, 1)
            parts.append(t)
        kern.renorm(d, i, 2, st["info"][3], None, st["site"], case["status"])       # names the output's blocks
        new = d.lenv[i] if left else d.renv[i + 1]
        out = torch.zeros_like(new.values)
        for (lay, off), t in zip(zip(new.layouts, new.offsets), parts):
            out[int(off):int(off) + lay.size] = _packed(lay, t)
        return out
    c = st["x"].reshape(len(d.qnuml[i]), 4, 4, -1)
    l, r = c.shape[0], c.shape[3]
    if case["status"] == "L":
        m = c.reshape(4 * l, 4 * r)
        out = m @ m.T
        for (el, ev), (wl, wv) in zip(_sets(L), _sets(W1)):
            t = torch.tensordot(_dense(el, ev), c.reshape(l, 4, 4 * r), ([2], [0]))             # a l n X
            t = torch.tensordot(_dense(wl, wv), t, ([0, 3], [0, 2])).permute(2, 1, 3, 0).reshape(4 * l, -1)
            out = out + NOISE * (t @ t.T)
        return out
    m = c.reshape(4 * l, 4 * r)
    out = m.T @ m
    for (el, ev), (wl, wv) in zip(_sets(R), _sets(W2)):
        t = torch.tensordot(c.reshape(4 * l, 4, r), _dense(el, ev), ([2], [2]))                 # Y n b r'
        t = torch.tensordot(_dense(wl, wv), t, ([1, 3], [2, 1])).permute(1, 3, 0, 2).reshape(4 * r, -1)
        out = out + NOISE * (t @ t.T)
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def _sec(q):
    s, n, _ = classification(q)
    return [(tuple(numpy.rint(2 * v).astype(int)), int(c)) for v, c in zip(s, n)]


def _fibers(bond_l, right, shift, sp):
    """Sum over (l, n1, n2, r) with q(l) - shift + q(n1) + q(n2) = q(r) of D_l D_r, by n1 and n2."""
    out = numpy.zeros((4, 4))
    rt = {}
    for q, c in right:
        rt[q[0] if sp else q] = rt.get(q[0] if sp else q, 0) + c
    ph = numpy.rint(2 * QPHYS).astype(int)
    for n1 in range(4):
        for n2 in range(4):
            for q, c in bond_l:
                t = tuple(numpy.array(q) - numpy.array(shift) + ph[n1] + ph[n2])
                out[n1, n2] += c * rt.get(t[0] if sp else t, 0)
    return out


def work(case):
    """Bytes: the environments, the two MPO sites and the vector or site tensor read once at
    the element size of the precision, the result written once.  Operations: two per
    non-zero product of the four (three) contractions in the reference's order, block pairs
    that symmetry allows, the MPO's non-zero elements only."""
    kind, K, D = case["kind"], case["K"], case["D"]
    N = nelec(K)
    if kind == "sweep":
        # one product, diagonal and renormalisation per dot: the least any solver does
        tot = {"bytes": 0.0, "flops": 0.0}
        for i in range(1, K - 2):
            for k in ("hvec", "hdiag", "renorm"):
                w = work({"kind": k, "K": K, "D": D, "site": i, "precision": "f64", "status": "R"})
                tot = {x: tot[x] + w[x] for x in tot}
        return tot
    i, sp = case["site"], kind == "sp"
    ql, qr = bond(K, N, i, D), bond(K, N, K - i - 2, D)
    left = _sec(ql)
    right = _sec(numpy.array([float(N), 0.0]) - qr)
    ham = make_hamiltonian(K, N, 1, DECAY)
    if sp:
        pts, _ = s2quad(case["npts"])
        m = build_mpo_sp(ham, pts, (i, i + 1))
    else:
        m = build_mpo(ham, (i, i + 1))
    el = 8 if case.get("precision", "f64") == "f64" else 4
    flops = 0.0
    nbytes = 0.0
    psi = _fibers(left, right, (0, 0), False)
    ndim0 = float(psi.sum())
    seen = {}
    for (l1, v1), (l2, v2) in zip(zip(*m[i]), zip(*m[i + 1])):
        key = (id(l1), id(l2))
        nz1, nz2 = _nonzero(l1, v1), _nonzero(l2, v2)
        if key not in seen:
            seen[key] = _class_work(left, right, l1, l2, sp)
        fib1, fib2, g1, g4, envl, envr = seen[key]
        if kind in ("hvec", "sp"):
            flops += g1 + g4 + 2 * float((nz1 * fib1[:, None, None, :]).sum()) + \
                2 * float((nz2 * fib2[:, None, None, :]).sum())
            nbytes += el * (envl + envr + len(v1) + len(v2))
        elif kind == "hdiag":
            z1, z2 = _neutral(l1, 0), _neutral(l2, 1)
            flops += 2.0 * 16 * z2 * (len(ql) * len(qr) / 8.0 + z1 * len(ql))
            nbytes += 8 * (z1 * len(ql) + z2 * len(qr))
        elif kind == "renorm":
            lft = case["status"] == "L"
            e, v, lay = (envl, v1, l1) if lft else (envr, v2, l2)
            sites = i + 1 if lft else K - i - 1
            new = len(bond(K, N, sites, D))
            old = len(ql) if lft else len(qr)
            # blocks of a site tensor: each old state meets about new/nsec of the new ones per physical state
            nsec = max(1, len(_sec(bond(K, N, sites, D))))
            flops += 2.0 * e * 4 * new / nsec * 2 + 2.0 * float((v != 0).sum()) * old * new / nsec
            nbytes += 8 * (e + len(v) + e * (new / float(max(1, old))) ** 2)
        else:
            lft = case["status"] == "L"
            flops += (g1 if lft else g4) + 2 * float(((nz1 * fib1[:, None, None, :]) if lft else
                                                     (nz2 * fib2[:, None, None, :])).sum())
            n = 4 * (len(ql) if lft else len(qr))
            flops += 2.0 * (n * n / 8.0) * ndim0 / n
            nbytes += 8 * (envl if lft else envr)
    if kind == "hvec":
        nbytes += 16 * ndim0
    elif kind == "sp":
        nbytes += 32 * ndim0
    elif kind == "hdiag":
        nbytes += 8 * ndim0
    elif kind == "prdm":
        n = 4 * (len(ql) if case["status"] == "L" else len(qr))
        nbytes += 8 * (ndim0 + n * n)
    return {"bytes": float(nbytes), "flops": float(flops)}


def _neutral(lay, index):
    """Extent of the MPO bond's sector of quantum number zero."""
    q = numpy.asarray(lay.qsyms[index])
    return float(numpy.asarray(lay.ndims[index])[(numpy.rint(2 * q) == 0).all(axis=1)].sum())


def _nonzero(lay, values):
    """Non-zero elements of W by (sector of its left bond, sector of its right bond, n', n)."""
    shape = [len(n) for n in lay.ndims]
    out = numpy.zeros(shape)
    tot = 0
    for k in range(4):
        q = numpy.rint(2 * numpy.asarray(lay.qsyms[k]))
        q = q.reshape((1,) * k + (len(q),) + (1,) * (3 - k) + (q.shape[-1],))
        tot = tot - q if lay.status[k] else tot + q
    o = 0
    for blk in numpy.argwhere((tot == 0).all(axis=-1)):
        n = int(numpy.prod([lay.ndims[k][s] for k, s in enumerate(blk)]))
        out[tuple(blk)] = numpy.count_nonzero(values[o:o + n])
        o += n
    return out


def _class_work(left, right, l1, l2, sp):
    """Fibers each MPO element of the two sites meets (by left bond sector and ket state), the
    products of L.psi and .R, and the elements of the two environments, for one operator class."""
    two = lambda q: (tuple(numpy.rint(2 * v).astype(int)) for v in q)                # noqa: E731
    a_sec = list(zip(two(l1.qsyms[0]), l1.ndims[0]))
    b_sec = list(zip(two(l1.qsyms[1]), l1.ndims[1]))
    c_sec = list(zip(two(l2.qsyms[1]), l2.ndims[1]))
    pad = lambda q: q if len(q) == 2 else (q[0], 0)                                   # noqa: E731
    fib1 = numpy.zeros((len(a_sec), 4))
    fib2 = numpy.zeros((len(b_sec), 4))
    g1 = g4 = envl = envr = 0.0
    psi_l = {}
    ph = numpy.rint(2 * QPHYS).astype(int)
    rd = dict(right)
    for q, c in left:
        psi_l[q] = sum(rd.get(tuple(numpy.array(q) + ph[n] + ph[m]), 0) for n in range(4) for m in range(4))
    for k, (qa, na) in enumerate(a_sec):
        f = _fibers(left, right, pad(qa), sp)
        fib1[k] = f.sum(axis=1)
        for q, c in left:
            for q2, c2 in left:
                ok = q2[0] == q[0] - qa[0] if sp else q2 == (q[0] - qa[0], q[1] - qa[1])
                if ok:
                    envl += na * c * c2
                    g1 += 2.0 * na * c * c2 * psi_l[q2]
    for k, (qb, nb) in enumerate(b_sec):
        fib2[k] = _fibers(left, right, pad(qb), sp).sum(axis=0)
    psi_r = {}
    ldim = dict(left)
    for q, c in right:
        psi_r[q] = sum(ldim.get(tuple(numpy.array(q) - ph[n] - ph[m]), 0) for n in range(4) for m in range(4))
    for qc, nc in c_sec:
        for q, c in right:
            for q2, c2 in right:
                ok = q[0] == q2[0] + qc[0] if sp else q == (q2[0] + qc[0], q2[1] + qc[1])
                if ok:
                    envr += nc * c * c2
                    g4 += 2.0 * nc * c * c2 * psi_r[q]
    return fib1, fib2, g1, g4, envl, envr
