"""The sparse two-site MPO stage (qc_wsparse): its records interpreted in NumPy against the
oracle-checked separate stages on the CPU, and the kernel against the grouped-GEMM sigma on
the GPU at the edges of its tiles (one fiber, 31 / 32 / 33, several sectors in one tile, 64
and 128 fibers, the last partial octet), in FP64, FP32 and split TF32."""
import numpy
import pytest
import torch

from helpers import load, layout_of, tensorset, record_operators
from emulate import patch_stage_run
from qcmpodmrg_b200 import engine
from qcmpodmrg_b200.hamiltonian import make_hamiltonian
from qcmpodmrg_b200.mpo import QPHYS, build_mpo
from qcmpodmrg_b200.qtensor import Layout, classification


def interpret(st, A, C, kind="f64"):
    """C written by the items of a SparseWStage, each element once, absent blocks zero."""
    a, c = A.numpy().astype(numpy.float64), C.numpy()
    hits = numpy.zeros(len(c), dtype=numpy.int64)
    for (tile, items, _, maxr, maxo) in st.items(kind):
        for it in items:
            d = st.h_deltas[it["delta"]]
            R = int(d["R"])
            assert 0 < it["nf"] <= tile and R <= maxr
            starts = st.h_groups["start"][d["grp_b"]:d["grp_e"]]
            pos = st.h_groups["start"][it["grp"]] + it["f0"] + numpy.arange(it["nf"])
            gi = numpy.searchsorted(starts, pos, side="right") - 1
            assert gi[0] + d["grp_b"] == it["grp"] and gi[-1] - gi[0] < engine.WX_GRPS
            f = pos - starts[gi]
            g = st.h_groups[d["grp_b"] + gi]
            assert (f < g["F"]).all()
            rows = st.h_rows[d["row_b"]:d["row_b"] + R]
            for op in range(it["op_b"], it["op_e"]):
                o = st.host_ops[op]
                T = numpy.zeros((R + 4, it["nf"]))
                for r, rec in enumerate(rows):
                    off = g["a"][:, rec >> 16]
                    ok = off >= 0
                    T[r, ok] = a[o["a_base"] + off[ok] + f[ok] + (rec & 0xffff) * g["F"][ok]]
                dop = st.h_dops[d["dop_b"] + op - it["op0"]]
                assert dop["noct"] <= maxo and dop["ent_b"] % 4 == 0
                for q in st.h_octs[dop["oct_b"]:dop["oct_b"] + dop["noct"]]:
                    e0, n = int(dop["ent_b"] + q["ent"]), int(q["cnt"])
                    assert n % 4 == 0
                    w = st.h_w[kind][8 * e0:8 * (e0 + n)]
                    # FP64: per step of four entries, lane l holds entry l % 4 and row l / 4
                    w = w.reshape(-1, 8, 4).transpose(0, 2, 1).reshape(-1, 8) if kind == "f64" else w.reshape(-1, 8)
                    val = w.T @ T[st.h_ent_r[e0:e0 + n]]                      # [8, nf]
                    for k, row in enumerate(q["row"]):
                        if row < 0:
                            assert not w[:, k].any()
                            continue
                        off = g["c"][:, row >> 16]
                        ok = off >= 0
                        dst = o["c_base"] + off + (f // g["flo"]) * g["h"][:, row >> 16] + f % g["flo"]
                        at = (dst + (row & 0xffff) * g["flo"])[ok]
                        hits[at] += 1
                        c[at] = val[k, ok]
    return hits


def interpret_panel(st, A, B, C):
    """C written by the units of a DPanelStage, each element once."""
    a, b, c = A.numpy(), B.numpy(), C.numpy()
    hits = numpy.zeros(len(c), dtype=numpy.int64)
    for w in st.h_work:
        u, o = st.h_units[w[0]], st.host_ops[w[1]]
        assert 0 < u["mrem"] <= engine.DP_TILE[st.kind][0] and 0 < u["nrem"] <= engine.DP_TILE[st.kind][1]
        assert (u["a_off"] + o["a_base"]) % 4 == 0 and (u["b_off"] + o["b_base"]) % 4 == 0 and u["lda"] % 4 == 0
        m, n, k = (numpy.arange(u[x]) for x in ("mrem", "nrem", "K"))
        blk = st.h_cols is None and st.h_crow is None
        am = a[o["a_base"] + u["a_off"] + (m[:, None] + k * u["lda"] if blk else m[:, None] * u["lda"] + k)]
        bm = b[o["b_base"] + u["b_off"] + n[:, None] * u["ldb"] + k]
        ok = numpy.ones(len(n), dtype=bool)
        if blk:
            dr, dc = (int(x) for x in u["pad"][:2])
            mm = u["m0"] + m[:, None]
            at = u["c_off"] + mm // dr * dr * dc + (u["n0"] + n) * dr + mm % dr
        elif st.h_cols is None:
            at = st.h_crow[u["c_off"] + m][:, None] + u["n0"] + n
        else:
            col = st.h_cols[u["c_off"] + n]
            ok = col["off"] >= 0
            at = col["off"].astype(numpy.int64) + (u["m0"] + m[:, None]) * col["ld"].astype(numpy.int64)
        at = (o["c_base"] + at)[:, ok]
        numpy.add.at(hits, at.ravel(), 1)
        c[at] = (o["alpha"] * (am @ bm.T))[:, ok]
    return hits


def patch(monkeypatch):
    patch_stage_run(monkeypatch)
    monkeypatch.setattr(engine.SparseWStage, "run",
                        lambda self, A, B, C, kind="f64", stream=None: interpret(self, A, C, kind))
    monkeypatch.setattr(engine.DPanelStage, "run", lambda self, A, B, C, stream=None: interpret_panel(self, A, B, C))



def sparse_sigma(r, device, sparse_w=True, precision="f64"):
    from qcmpodmrg_b200.kernels import SigmaOperator, Workspace
    opers = [int(x) for x in numpy.atleast_1d(r["opers"])]
    return SigmaOperator(Workspace(torch.device(device)), int(r["key"][2]), layout_of(r["qtmp"]),
                         tensorset(r["envL"], device), tensorset(r["envR"], device), tensorset(r["mpo_i"], device),
                         tensorset(r["mpo_j"], device), numpy.asarray(r["qkey"], dtype=numpy.float64), opers,
                         numpy.atleast_1d(r["hpwts"]).astype(numpy.float64), precision, use_fiber=True, fuse_w=False,
                         sparse_w=sparse_w)


@pytest.mark.parametrize("tag", ["K4", "K5", "K6", "K5N2"])
def test_sparse_records_reproduce_the_separate_stages(tag, monkeypatch):
    """T3 of the sparse records equals T3 of the two separate stages, every element of the
    T3 panels that stage writes is written exactly once, and sigma is the reference's."""
    patch(monkeypatch)
    used = 0
    for r in load("kernels_%s.npz" % tag)["records"]:
        sig = sparse_sigma(r, "cpu", precision="f32")
        x = torch.from_numpy(numpy.asarray(r["hvec_x"], dtype=numpy.float64))
        ref = numpy.asarray(r["hvec_y"])
        assert numpy.abs(sig(x, precision="f64").numpy() - ref).max() <= 1e-12 * max(1.0, numpy.abs(ref).max())
        if sig.wx is None:
            continue
        used += 1
        T1 = torch.zeros(sig.tot[0] + 64, dtype=torch.float64)
        T2 = torch.zeros(sig.tot[1] + 64, dtype=torch.float64)
        psi = torch.zeros(sig._psi_total, dtype=torch.float64)
        from qcmpodmrg_b200 import kernels
        kernels.gather_pad(x, sig._psi_gidx, psi)
        hits = interpret_panel(sig.d1, sig.lpan64, psi, T1)
        T0 = torch.zeros_like(T1)
        sig._stages[0].run(sig.a1("f64"), x, T0, "f64")
        assert hits.max() == 1 and numpy.abs((T1 - T0).numpy()).max() <= 1e-13 * max(1.0, T0.abs().max().item())
        ta, tb = torch.zeros(sig.tot[2] + 64, dtype=torch.float64), torch.zeros(sig.tot[2] + 64, dtype=torch.float64)
        sig.stages[1].run(T1, sig.Wi.values, T2, "f64")         # the stages compiled on demand
        sig.stages[2].run(T2, sig.Wj.values, tb, "f64")
        for kind, tol in (("f64", 1e-13), ("f32", 1e-6)):
            ta.zero_()
            hits = interpret(sig.wx, T1, ta, kind)
            assert hits.max() <= 1
            assert numpy.abs(ta.numpy() - tb.numpy()).max() <= tol * max(1.0, tb.abs().max().item())
            assert (hits[tb.numpy() != 0] == 1).all()
        part = torch.zeros(sig.nops * sig.ndim0, dtype=torch.float64)
        ref4 = torch.zeros_like(part)
        assert interpret_panel(sig.d4, tb, sig.rpan64, part).max() == 1
        sig._stages[3].run(tb, sig.b4("f64"), ref4, "f64")
        assert numpy.abs((part - ref4).numpy()).max() <= 1e-13 * max(1.0, ref4.abs().max().item())
        # the FP32 panels: the same elements, each once; operands rounded to 2^-24, sums below 2^5 terms
        for st, a, b, out in ((sig.f1, sig.lpan_f32, psi, T0), (sig.f4, tb, sig.rpan_f32, ref4)):
            c = torch.zeros_like(out)
            assert interpret_panel(st, a, b, c).max() == 1
            assert numpy.abs((c - out).numpy()).max() <= 1e-5 * max(1.0, out.abs().max().item())


@pytest.mark.parametrize("tag", ["SP_K4", "SP_K5"])
def test_sparse_plan_of_the_spin_projected_operators(tag, monkeypatch):
    """N-only quantum numbers, blocks outside the (N, Sz) wavefunction left out: H and S
    products equal those of the separate stages."""
    from helpers import record_sp_operators
    from qcmpodmrg_b200 import kernels
    patch(monkeypatch)
    used = 0
    for r in load("kernels_%s.npz" % tag)["records"]:
        ref = record_sp_operators(r, "cpu")
        make = kernels.SigmaOperator.__init__
        with monkeypatch.context() as m:
            m.setattr(kernels.SigmaOperator, "__init__",
                      lambda self, *a, **k: make(self, *a, **dict(k, sparse_w=True)))
            new = record_sp_operators(r, "cpu")
        for a, b in zip(ref[:2], new[:2]):
            used += b.inner.wx is not None
            x = torch.from_numpy(numpy.random.default_rng(1).standard_normal(a.ndim0))
            ya, yb = a(x).numpy(), b(x).numpy()
            assert numpy.abs(ya - yb).max() <= 1e-12 * max(1.0, numpy.abs(ya).max())
    assert used
    assert used


@pytest.mark.parametrize("tag", ["K4", "K5", "K6", "K5N2", "SP_K4", "SP_K5"])
def test_panel_renormalisation_matches_the_grouped_one(tag, monkeypatch):
    """Both directions: the same layouts, and values within rounding of the grouped block GEMM.
    Spin projection's N-only site tensors sum several blocks into one intermediate: they keep
    the grouped form."""
    from helpers import record_renormalizer, record_sp_renormalizers
    from qcmpodmrg_b200 import kernels
    patch(monkeypatch)
    rec = (lambda r: record_sp_renormalizers(r, "cpu")) if tag.startswith("SP") else \
        (lambda r: (lambda x: (x[0], x[1]))(record_renormalizer(r, "cpu")))
    used = 0
    make = kernels.Renormalizer.__init__
    for r in load("kernels_%s.npz" % tag)["records"]:
        if "renorm_site" not in r:
            continue
        ref = rec(r)
        with monkeypatch.context() as m:
            m.setattr(kernels.Renormalizer, "__init__", lambda self, *a: make(self, *a, panels=True))
            new = rec(r)
        site = torch.from_numpy(ref[-1])
        for a, b in zip(ref[:-1], new[:-1]):
            used += b.ep is not None
            ea, eb = a(site), b(site)
            for i in range(len(ea.layouts)):
                assert eb.layouts[i] is ea.layouts[i]
                va, vb = ea.op_values(i).numpy(), eb.op_values(i).numpy()
                assert numpy.abs(va - vb).max() <= 1e-13 * max(1.0, numpy.abs(va).max())
    assert bool(used) != tag.startswith("SP")


@pytest.mark.parametrize("tag", ["NZ_K5", "NZ_K6", "NZSP_K5"])
def test_panel_noise_term_matches_the_grouped_one(tag, monkeypatch):
    """Both directions: the dense noise matrix within rounding of the grouped block GEMM's."""
    from helpers import record_noise
    from qcmpodmrg_b200 import kernels
    patch(monkeypatch)
    used = 0
    make = kernels.NoiseRDM.__init__
    for r in load("kernels_%s.npz" % tag)["records"]:
        if "prdm_cimat" not in r:
            continue
        ref, vals, _ = record_noise(r, "cpu")
        with monkeypatch.context() as m:
            m.setattr(kernels.NoiseRDM, "__init__", lambda self, *a: make(self, *a, panels=True))
            new = record_noise(r, "cpu")[0]
        used += new.ep is not None
        a, b = ref(vals).numpy(), new(vals).numpy()
        assert a.shape == b.shape and numpy.abs(a - b).max() <= 1e-13 * max(1.0, numpy.abs(a).max())
    assert bool(used) != ("SP" in tag)


def test_changed_mpo_values_are_seen():
    """The host copy of a TensorSet is not used once the device values were changed in place."""
    from qcmpodmrg_b200.kernels import TensorSet
    r = load("kernels_K4.npz")["records"][0]
    w = tensorset(r["mpo_i"], "cpu")
    assert w.host() is w.host()
    w.values[0] += 1.0
    assert w.host()[0] == float(w.values[0])
    w2 = TensorSet(w.layouts, w.values.clone(), w.offsets)
    assert numpy.array_equal(w2.host(), w.host())


def _dot(K, isite, nl, nr, dev, precision, seed=0, sparse_w=None):
    """A dot whose bonds have the given states per (N, Sz) sector, with random environments."""
    from qcmpodmrg_b200.kernels import SigmaOperator, TensorSet, Workspace
    N = K
    ham = make_hamiltonian(K, N, 3, 3.0)
    W = {i: TensorSet(*v, device=dev) for i, v in build_mpo(ham, (isite, isite + 1)).items()}
    ql = numpy.array([[n, 0.5 * s] for n, s, c in nl for _ in range(c)])
    qr = numpy.array([[n, 0.5 * s] for n, s, c in nr for _ in range(c)])
    qkey = numpy.array([float(N), 0.0])
    cl = [classification(q) for q in (ql, QPHYS, QPHYS, qkey - qr)]
    psi = Layout([False, False, False, True], [c[0] for c in cl], [c[1] for c in cl])
    gen = torch.Generator(device="cpu").manual_seed(seed)

    def env(lays, k, sign, q):
        c = classification(q)
        out = [Layout([True, False, True], [sign * l.qsyms[k], c[0], c[0]], [l.ndims[k], c[1], c[1]]) for l in lays]
        v = torch.randn(sum(l.size for l in out), dtype=torch.float64, generator=gen).to(dev)
        return TensorSet(out, v, device=dev)

    L, R = env(W[isite].layouts, 0, 1.0, ql), env(W[isite + 1].layouts, 1, -1.0, qr)
    opers = list(range(2 * K))
    mk = lambda **kw: SigmaOperator(Workspace(torch.device(dev)), isite, psi, L, R, W[isite], W[isite + 1], qkey,  # noqa: E731
                                    opers, numpy.ones(2 * K), precision, **kw)
    x = torch.randn(psi.size, dtype=torch.float64, generator=gen).to(dev)
    return mk, x


SECTORS = [
    ([(3, 1, 1), (4, 0, 1), (5, -1, 1)], [(3, 1, 1), (4, 0, 1), (3, -1, 1)]),             # one fiber per sector pair
    ([(4, 0, 31), (3, 1, 1), (5, 1, 1)], [(4, 0, 1), (3, -1, 1), (3, 1, 1)]),             # 31 fibers
    ([(4, 0, 8), (3, -1, 3), (5, 1, 2)], [(4, 0, 4), (3, 1, 11), (2, 0, 3)]),             # 32 and 33 fibers
    ([(4, 0, 13), (3, -1, 7), (3, 1, 5), (5, -1, 6), (2, 0, 2), (6, 0, 3)],
     [(4, 0, 10), (3, 1, 9), (3, -1, 6), (5, 1, 4), (2, 0, 3)]),                          # several tiles, ragged
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(SECTORS)))
@pytest.mark.parametrize("precision", ["f64", "f32", "tf32x3"])
def test_kernel_at_the_edges_of_its_tiles(case, precision, cuda, monkeypatch):
    """FP64 within 1e-12 of the grouped GEMM, FP32 within 2e-5, at every fiber-tile width
    (the shared-memory budget forces 32, 64 and 128 fibers)."""
    nl, nr = SECTORS[case]
    mk, x = _dot(8, 3, nl, nr, cuda, precision)
    ref = mk(use_fiber=False, panel1=False)(x, precision="f64").cpu().numpy()
    monkeypatch.setattr(engine, "WX_SMALL", 0)
    for budget in (1, 40 * 1024, 100 * 1024):
        monkeypatch.setattr(engine, "WX_TILE_BYTES", budget)
        sig = mk(use_fiber=True, fuse_w=False)
        assert sig.wx is not None
        y = sig(x).cpu().numpy()
        if precision == "f64":
            assert numpy.abs(y - ref).max() <= 1e-12 * numpy.abs(ref).max(), budget
        else:
            assert numpy.linalg.norm(y - ref) <= 2e-5 * numpy.linalg.norm(ref), budget
        assert numpy.array_equal(y, sig(x).cpu().numpy())
