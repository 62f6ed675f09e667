"""Device operators of the two-site hot path: sigma, diagonal, renormalisation.

  SigmaOperator  <- HVecQt        source/mpo_dmrg_kernelQt.py:153-319 (two-site :238-317)
  DiagOperator   <- HDiagQt       source/mpo_dmrg_kernelQt.py:30-127  (two-site :77-119)
  Renormalizer   <- renormQt_H00  source/mpo_dmrg_kernelQt.py:633-767 (also genHopsQt,
                                  source/mpo_dmrg_initQt.py:88-271, which is the same chain)

The reference loops over operators p, MPO slices and block pairs in Python and
calls numpy.tensordot per pair.  Here the operator loop is folded into the
work lists: each of the four sigma contractions (L.psi, .W_i, .W_{i+1}, .R) is
one launch over all operators and all block pairs, with intermediates in HBM
scratch and the sum over operators done inside the last launch (no atomics).
Block-pair lists are built per symmetry class of the operator, as the
reference caches its templates per class.
"""
import ctypes

import numpy
import torch

from . import native
from .native import check
from .engine import (Stage, compile_classes, add_parts, live_blocks, prune, op_table, TASK_DT, CONTRIB_DT, LOG,
                     compile_fiber, FiberStage, CompositeStage, panel_sigma1, compile_panels, BPERM_DT, PanelStage,
                     fiber_stages, panel_sigma4, upload, sparse_w_class, SparseWStage,
                     DPanelStage, dpanel_units, DCOL_DT, psi_panels, WSource, transposed_values, _ranges)
from .envpanels import EnvPanels, NoPanelForm
from .mpo import case
from .qtensor import Contraction, Layout, flip_right, flip_horizontal


class Workspace(object):
    """Grow-only device scratch buffers shared by all operators of a context."""

    def __init__(self, device):
        self.device = device
        self.bufs = {}

    def get(self, name, numel, dtype):
        b = self.bufs.get((name, dtype))
        if b is None or b.numel() < numel:
            self.bufs.pop((name, dtype), None)
            b = torch.empty(max(int(numel), 1) + 64, dtype=dtype, device=self.device)
            self.bufs[(name, dtype)] = b
        return b


class TensorSet(object):
    """Per-operator block tensors (environments or site operators) back to back in one buffer."""

    def __init__(self, layouts, values, offsets=None, device=None):
        self.layouts = list(layouts)
        if offsets is None:
            sizes = numpy.array([l.size for l in self.layouts], dtype=numpy.int64)
            offsets = numpy.concatenate([[0], numpy.cumsum(sizes)[:-1]]).astype(numpy.int64)
        self.offsets = numpy.asarray(offsets, dtype=numpy.int64)
        self.total = int(self.offsets[-1] + self.layouts[-1].size) if self.layouts else 0
        if isinstance(values, (list, tuple)):
            host = numpy.concatenate([numpy.asarray(v, dtype=numpy.float64) for v in values]) \
                if values else numpy.zeros(0)
            ref = torch.from_numpy(host).to(device)
            values = ref.clone()
            self._given = (host, ref)               # what host() compares the values with
        else:
            self._given = None
        self.values = values
        self._f32 = None
        self._finite = self._transposed = None

    def f32(self):
        if self._f32 is None or self._f32.data_ptr() == 0:
            self._f32 = self.values.to(torch.float32)
        return self._f32

    def host(self, check=True):
        """The values as a host array.  Those the set was made from serve while the device values
        equal them: compared on the device at every call, as a collective, a native kernel or a
        write through ``.data`` changes values without a trace on the tensor (K=24: 5 MB a site,
        a comparison instead of a copy); otherwise a copy from the device.  Both wait for the
        stream.  check=False: as last found, for a caller that compares later (EnvPanels.current)."""
        if self._given is not None:
            host, ref = self._given
            v = self.values
            if not check or (v.device == ref.device and v.dtype == ref.dtype and torch.equal(v, ref)):
                return host
            self._given = None
        return self.values.detach().to("cpu", torch.float64, copy=True).numpy()

    def finite(self, host):
        """Whether every element of ``host``, an array that host() returned, is finite.  The sparse
        MPO stage needs that: it multiplies T1 blocks that symmetry leaves out as zeros, and drops
        zero products."""
        if self._finite is None or self._finite[0] is not host:
            self._finite = (host, bool(numpy.isfinite(host).all()))
        return self._finite[1]

    def transposed(self, host):
        """``host``, an array that host() returned, with the bonds of every block exchanged: made
        once for an array (K=24: 2 to 4 ms, which every renormalisation and noise term from the right
        paid)."""
        if self._transposed is None or self._transposed[0] is not host:
            self._transposed = (host, transposed_values(self.layouts, host, self.offsets))
        return self._transposed[1]

    def op_values(self, i):
        o = int(self.offsets[i])
        return self.values[o:o + self.layouts[i].size]

    def nbytes(self):
        return self.values.numel() * self.values.element_size()


def _stream(device):
    return torch.cuda.current_stream(device).cuda_stream


def block_permute(descs, ndescs, opspan, ops, src, dst):
    """Per-dot block permutation of an FP64 tensor set into dst (FP64 or FP32), qc_block_permute."""
    check(native.lib().qc_block_permute(descs.data_ptr(), ndescs, opspan, ops.data_ptr(), src.data_ptr(),
                                        dst.data_ptr(), int(dst.dtype == torch.float32), _stream(dst.device)),
          "qc_block_permute")
    LOG.launches += 1
    return dst


def gather(src, idx, out):
    """out[i] = src[idx[i]] on the device (qc_gather_f64)."""
    check(native.lib().qc_gather_f64(src.data_ptr(), idx.data_ptr(), out.data_ptr(), out.numel(),
                                     _stream(out.device)), "qc_gather_f64")
    LOG.launches += 1
    return out


def scatter(src, idx, out):
    """out = 0; out[idx[i]] = src[i] on the device (qc_scatter_f64)."""
    check(native.lib().qc_scatter_f64(src.data_ptr(), idx.data_ptr(), out.data_ptr(), idx.numel(), out.numel(),
                                      _stream(out.device)), "qc_scatter_f64")
    LOG.launches += 1
    return out


def convert(src, out):
    """FP64 <-> FP32 conversion on the device."""
    lib = native.lib()
    n = min(src.numel(), out.numel())
    if src.dtype == torch.float64:
        check(lib.qc_convert_f64_to_f32(src.data_ptr(), out.data_ptr(), n, _stream(out.device)), "convert")
    else:
        check(lib.qc_convert_f32_to_f64(src.data_ptr(), out.data_ptr(), n, _stream(out.device)), "convert")
    LOG.launches += 1
    return out


def gather_split(x, idx, hi, lo):
    """hi[i] = tf32(x[idx[i]]), lo[i] = tf32(x[idx[i]] - hi[i]); idx < 0 gives 0 (qc_gather_split_f32)."""
    check(native.lib().qc_gather_split_f32(x.data_ptr(), idx.data_ptr(), idx.numel(), hi.data_ptr(), lo.data_ptr(),
                                           _stream(hi.device)), "qc_gather_split_f32")
    LOG.launches += 1
    return hi, lo


def gather_pad(x, idx, out):
    """out[i] = x[idx[i]] in out's type, 0 where idx is negative (qc_gather_pad_f64, _f32)."""
    if out.device.type != "cuda":           # plans interpreted on the CPU
        out[:idx.numel()] = torch.where(idx >= 0, x[idx.clamp(min=0)], torch.zeros((), dtype=x.dtype))
        return out
    fn = native.lib().qc_gather_pad_f64 if out.dtype == torch.float64 else native.lib().qc_gather_pad_f32
    check(fn(x.data_ptr(), idx.data_ptr(), idx.numel(), out.data_ptr(), _stream(out.device)), "qc_gather_pad")
    LOG.launches += 1
    return out


def tf32_split(hi, lo):
    """hi = tf32(x), lo = tf32(x - hi) for the FP32 values x held in hi (qc_tf32_split)."""
    check(native.lib().qc_tf32_split(hi.data_ptr(), lo.data_ptr(), hi.numel(), _stream(hi.device)),
          "qc_tf32_split")
    LOG.launches += 1
    return hi, lo


def reduce_ops(part, nops, n, out):
    """out = sum over operators of the per-operator partial vectors (qc_reduce_ops_*)."""
    lib = native.lib()
    fn = lib.qc_reduce_ops_f64 if part.dtype == torch.float64 else lib.qc_reduce_ops_f32
    check(fn(part.data_ptr(), nops, n, out.data_ptr(), _stream(out.device)), "qc_reduce_ops")
    LOG.launches += 1
    return out


def _groups(opers, isite, ncsite):
    g = {}
    for iop, p in enumerate(opers):
        g.setdefault(case(p, isite, ncsite), []).append(iop)
    return g


def _ncols(c, triples):
    """N extent (product of the operand-2 external dims) of the output blocks a stage writes."""
    if len(triples) == 0:
        return numpy.array([64])
    ne1 = c.l1.rank - len(c.axes[0])
    ob = numpy.unique(triples[:, 0])
    return numpy.prod(c.out.block_dims(ob)[:, ne1:], axis=1)


def unit_phys_t2(lay):
    """True when every block of the intermediate T2 = T1 . W_i, axes (l', n2, r, b, n1'),
    has extent 1 on its two physical axes (1 and 4)."""
    if lay.rank != 5 or len(lay.idx_allowed) == 0:
        return False
    d = lay.block_dims(lay.idx_allowed)
    return bool(numpy.all(d[:, 1] == 1) and numpy.all(d[:, 4] == 1))


def pair_flops(c, t):
    """2*M*N*K summed over the block pairs of one contraction (one operator)."""
    if len(t) == 0:
        return 0.0
    ne1 = c.l1.rank - len(c.axes[0])
    d = c.out.block_dims(t[:, 0]).astype(numpy.float64)
    k = c.l1.block_dims(t[:, 1])[:, c.axes[0]].astype(numpy.float64)
    return 2.0 * float((d.prod(axis=1) * k.prod(axis=1)).sum())


class SigmaOperator(object):
    """sigma = sum_p w_p R_p W_p[i+1] W_p[i] L_p psi for the dot (isite, isite+1)."""

    def __init__(self, ws, isite, psi_layout, L, R, Wi, Wj, qkey, opers, hpwts, precision="f64",
                 tensor_cores=None, use_fiber=False, fuse_w=True, panel1=True, panel4=True, live=None,
                 fg_budget=None, sparse_w=None, direct=True):
        """direct: the K-major panels of a product on its own are made now; False: by the first such
        product (lockstep batches run on the row-major panels and would hold both).
        sparse_w: the two MPO-site contractions as one sparse product (qc_wsparse, the fiber
        path without fuse_w); None: on a GPU, where the plan's blocks allow it.
        fg_budget: (A, W) shared-memory budgets of the dense fiber-group GEMM (qc_fgemm), as
        chosen by qcmpodmrg_b200.autotune; None keeps the engine's defaults.
        live: optional mask over the wavefunction layout's flat blocks.  Blocks outside it
        are zero in every input vector and discarded in every output (the blocks that N
        symmetry adds to an (N, Sz) wavefunction under spin projection): block pairs that
        read them in the first contraction or write them in the last are not compiled."""
        self.ws, self.psi, self.precision = ws, psi_layout, precision
        # tcgen05 tiles for the two large contractions (L.psi and .R) in TF32 modes
        tc = (precision in ("tf32", "tf32x3")) if tensor_cores is None else tensor_cores
        # tf32x3: the .R panel GEMMs on the TMA-fed tcgen05 kernel (qc_tcpanel_f32); the older
        # gathered tensor-core tiles (qc_bgemm_tf32*) stay for plain tf32 and explicit requests
        want_tc4 = precision == "tf32x3" and tensor_cores is None and use_fiber and panel4
        want_tc1 = precision == "tf32x3" and tensor_cores is None and panel1
        if want_tc4 or want_tc1:
            tc = False
        self.L, self.R, self.Wi, self.Wj = L, R, Wi, Wj
        self._lays = (list(L.layouts), list(R.layouts))      # held: identity is the plan's key
        dev = ws.device
        groups = _groups(opers, isite, 2)
        nops = len(opers)
        ax = (([2], [0]), ([0, 2], [0, 3]), ([1, 3], [3, 0]), ([1, 3], [2, 0]))
        bases = [numpy.zeros(nops, dtype=numpy.int64) for _ in range(3)]
        tot = [0, 0, 0]
        wbase = numpy.zeros(nops, dtype=numpy.int64)
        wtot = 0
        plans = {}
        self._fiber_args = (ax, groups, qkey, live, fg_budget)
        if sparse_w is None:
            sparse_w = torch.device(dev).type == "cuda"
        sparse_w = bool(sparse_w) and use_fiber and not fuse_w and panel1 and panel4
        chains, sx = {}, {}
        for key, ops in sorted(groups.items()):
            i0 = ops[0]
            Ll, W1, W2 = L.layouts[i0], Wi.layouts[i0], Wj.layouts[i0]
            Rl = flip_right(R.layouts[i0], qkey)
            for i in ops:
                if (L.layouts[i] is not Ll or Wi.layouts[i] is not W1 or Wj.layouts[i] is not W2
                        or flip_right(R.layouts[i], qkey) is not Rl):
                    raise ValueError("operators of one symmetry class must share their block structure")
            chains[key] = ch = self._chain(Ll, W1, W2, Rl, use_fiber, panel1, panel4, sparse_w)
            if sparse_w:
                (c1, t1), _, (c3, _), _, pan, pan4 = ch
                sx[key] = sparse_w_class(c1, t1, pan["t1off"], c3.out, pan4, W1, W2, psi_layout) \
                    if pan is not None and pan4 is not None else None
                sparse_w = sx[key] is not None
        for key, ops in sorted(groups.items()):
            i0 = ops[0]
            W1, W2 = Wi.layouts[i0], Wj.layouts[i0]
            Rl = flip_right(R.layouts[i0], qkey)
            if sx and not sparse_w:         # a class has no sparse form: the separate stages' T3 order
                chains[key] = self._chain(L.layouts[i0], W1, W2, Rl, use_fiber, panel1, panel4)
            (c1, t1), (c2, t2), (c3, t3), (c4, t4all), pan, pan4 = chains[key]
            t1off = pan["t1off"] if pan is not None else None
            # .W_i and .W_{i+1} fused: T3 = T1 . (W_i W_{i+1}) with the two-site MPO
            # block Wij[a, n1', n1, c, n2', n2] = sum_b W_i[a, b, n1', n1] W_{i+1}[b, c, n2', n2]
            # made once per dot, so T2 is never written (fiber-group kernel only)
            o3 = {} if pan4 is None else {"out_off": pan4["t3off"], "out_fhs": pan4["t3fhs"],
                                          "out_flo": pan4["t3flo"], "extra_out": pan4["needed"]}
            fused = None
            fib2 = fib3 = None
            if use_fiber and fuse_w:
                cW = Contraction(W1, W2, ([1], [0]))
                cF = Contraction(c1.out, cW.out, ([0, 2, 3], [0, 2, 5]))
                if cF.out is c3.out:
                    tF = prune(cF.triples, live1=live_blocks(c1.out, t1), live2=live_blocks(cW.out, cW.triples))
                    fp = compile_fiber(cF, tF, 0, 0, in_off=t1off, **o3)
                    if fp is not None:
                        fused = (cW, cF, tF, fp)
            elif use_fiber and not sparse_w:
                fib2, fib3 = self._fiber_pair(c1, c2, t2, c3, t3, t1off, o3)
                if fib3 is None and pan4 is not None:
                    pan4 = None
                    fib2, fib3 = self._fiber_pair(c1, c2, t2, c3, t3, t1off, {})
            if pan4 is not None and fused is None and fib3 is None and not sparse_w:
                pan4 = None                 # T3 comes from the grouped GEMM in the packed layout
            t4 = prune(t4all, live1=live_blocks(c3.out, fused[2] if fused else t3))
            if c4.out is not psi_layout:
                raise ValueError("sigma output layout differs from the wavefunction template")
            plans[key] = (ops, (c1, t1), (c2, t2), (c3, t3), (c4, t4), Rl, fused, pan, pan4, fib2, fib3)
            for s, c in enumerate((c1, c2, c3)):
                if s == 1 and fused is not None:
                    continue            # no T2 for fused classes
                size = pan["t1size"] if (s == 0 and pan is not None) else c.out.size
                if s == 2 and pan4 is not None:
                    size = pan4["t3size"]
                size = (int(size) + 31) // 32 * 32      # 128-byte aligned operator slices (TMA)
                for i in ops:
                    bases[s][i] = tot[s]
                    tot[s] += size
            if fused is not None:
                for i in ops:
                    wbase[i] = wtot
                    wtot += fused[0].out.size
        self.tot = tot
        self.nops = nops
        hp = numpy.asarray(hpwts, dtype=numpy.float64)
        # operator tables: operators ordered class by class; the last contraction
        # writes one partial sigma per operator (slot = position in that order)
        order = numpy.concatenate([numpy.array(plans[k][0]) for k in sorted(plans)])
        slot = numpy.arange(nops, dtype=numpy.int64) * psi_layout.size
        tabs = [op_table(L.offsets[order], 0, bases[0][order], 1.0),
                op_table(bases[0][order], Wi.offsets[order], bases[1][order], 1.0),
                op_table(bases[1][order], Wj.offsets[order], bases[2][order], 1.0),
                op_table(bases[2][order], R.offsets[order], slot, hp[order])]
        st = [{}, {}, {}, {}]
        fib = [[], [], [], []]
        fuse_parts, wij_parts = [], {}
        wx_parts = []
        # how the W contractions of each symmetry class run: sparse product / fused / fiber /
        # grouped GEMM
        self.w_paths = {"sparse": 0, "fused": 0, "fiber": 0, "generic": 0}
        pos = 0
        # W contractions: fiber-group kernel (inputs staged once per fiber tile) where
        # every group fits in shared memory, generic grouped GEMM otherwise
        lperm = []
        pst, pst_tc = {}, {}            # panel GEMM parts of the L.psi contraction
        rperm = []
        p4st, p4st_tc = {}, {}          # panel GEMM parts of the .R contraction
        crow_all, crow_n = [], 0        # their row table (panel row -> sigma element offset)
        tc4_classes = []                # (operator range, pan4, row-table base) for the tensor-core .R
        tc1_classes = []                # (operator range, pan["tc"]) for the tensor-core L.psi
        any4 = any(v[8] is not None for v in plans.values())
        for key, (ops, *cs, Rl, fused, pan, pan4, fib2, fib3) in sorted(plans.items()):
            rng = (pos, pos + len(ops))
            pos += len(ops)
            t1off = pan["t1off"] if pan is not None else None
            if panel1:
                if pan is not None:
                    src, dst, n = pan["lperm"]
                else:                   # no panels for this class: L blocks copied in place
                    Ll = cs[0][0].l1
                    src = dst = Ll.ioff[Ll.idx_allowed]
                    n = Ll.ndim[Ll.idx_allowed]
                d = numpy.zeros(len(src), BPERM_DT)
                d["src_off"], d["dst_off"] = src, dst
                d["d0"], d["d1"], d["d2"] = 1, 1, n
                d["s2"] = 1
                d["op_b"], d["op_e"] = rng
                lperm.append(d)
            if any4:
                d = numpy.zeros(0, BPERM_DT)
                if pan4 is not None:
                    src, dst, dU, st3 = pan4["rperm"]
                    d = numpy.zeros(len(src), BPERM_DT)
                    d["src_off"], d["dst_off"] = src, dst
                    d["d0"], d["d1"], d["d2"] = dU[:, 0], dU[:, 1], dU[:, 2]
                    d["s0"], d["s1"], d["s2"] = st3
                else:                       # R blocks copied in place
                    src = dst = Rl.ioff[Rl.idx_allowed]
                    d = numpy.zeros(len(src), BPERM_DT)
                    d["src_off"], d["dst_off"] = src, dst
                    d["d0"], d["d1"], d["d2"] = 1, 1, Rl.ndim[Rl.idx_allowed]
                    d["s2"] = 1
                d["op_b"], d["op_e"] = rng
                rperm.append(d)
            if pan4 is not None:
                g4 = pan4["gemm"]
                g4 = g4[:6] + (g4[6] + crow_n,) + tuple(g4[7:])     # row-table indices into the stage's table
                if want_tc4 or sparse_w:
                    tc4_classes.append((rng, pan4, crow_n))
                crow_all.append(pan4["crow"])
                crow_n += len(pan4["crow"])
                parts = compile_panels(g4, rng, tensor_cores=bool(tc))
                if tc:
                    parts, tcp = parts
                    add_parts(p4st_tc, tcp)
                for cfg, part in parts.items():
                    p4st.setdefault(cfg, []).append(part)
            if sparse_w:
                wx_parts.append((sx[key], ops, rng))
                self.w_paths["sparse"] += 1
            if fib3 is not None:
                fib[2].append(fib3 + (rng,))
                self.w_paths["fiber"] += 1
            if fused is not None:
                cW, cF, tF, fp = fused
                fuse_parts.append(fp + (rng,))
                self.w_paths["fused"] += 1
                add_parts(wij_parts, compile_classes(cW, cW.triples, ([1], [0])), op_range=rng)
            for si, (c, t) in enumerate(cs):
                if fused is not None and si in (1, 2):
                    continue
                if (si == 2 and fib3 is not None) or (si == 3 and pan4 is not None):
                    continue
                if si == 0 and pan is not None:
                    if want_tc1 or sparse_w:
                        tc1_classes.append((rng, pan["tc"]))
                    parts = compile_panels(pan["gemm"], rng, tensor_cores=bool(tc))
                    if tc:
                        parts, tcp = parts
                        add_parts(pst_tc, tcp)
                    for cfg, part in parts.items():
                        pst.setdefault(cfg, []).append(part)
                    continue
                off1 = t1off if si == 1 else None
                if si == 1 and fib2 is not None:
                    fib[1].append(fib2 + (rng,))
                    self.w_paths["fiber"] += 1
                    continue
                if sparse_w and si in (1, 2):
                    continue
                if si in (1, 2):
                    self.w_paths["generic"] += 1
                add_parts(st[si], compile_classes(c, t, ax[si], tensor_cores=tc if si in (0, 3) else False,
                                                  off1=off1), op_range=rng)
        self._stages = []
        self._tabs = tabs
        for si in range(4):
            if sparse_w and si in (1, 2):
                self._stages.append(None)       # compiled when the stage list is asked for
                continue
            g = Stage(st[si], dev, "sigma%d" % (si + 1), tabs[si]) if st[si] else None
            f = fiber_stages(fib[si], dev, "sigma%d" % (si + 1), tabs[si], fg_budget) if fib[si] else []
            if si == 0:
                self._s0_generic = g
            if si == 0 and (pst or pst_tc):
                f = [PanelStage(pst, dev, "sigma1", tabs[0], pst_tc)]
            if si == 3 and (p4st or p4st_tc):
                f = [PanelStage(p4st, dev, "sigma4", tabs[3], p4st_tc,
                                crow=numpy.concatenate(crow_all) if crow_all else None)]
            if not f:
                self._stages.append(g if g is not None else Stage({}, dev, "sigma%d" % (si + 1), tabs[si]))
            else:
                self._stages.append(CompositeStage(f + [g], "sigma%d" % (si + 1)))
        # the two MPO-site contractions as one sparse product, T1 -> T3
        self.wx = None
        self._plans, self._part_full = {}, False
        if sparse_w:
            w1, w2 = Wi.host(), Wj.host()
            if not (Wi.finite(w1) and Wj.finite(w2)):
                self.__init__(ws, isite, psi_layout, L, R, Wi, Wj, qkey, opers, hpwts, precision, tensor_cores,
                              use_fiber, fuse_w, panel1, panel4, live, fg_budget, sparse_w=False, direct=direct)
                return
            parts = [(x, rng, (WSource.of(x["W"][0], w1, Wi.offsets[ops]), WSource.of(x["W"][1], w2, Wj.offsets[ops])))
                     for x, ops, rng in wx_parts]
            self.wx = SparseWStage(parts, dev, "sigma23", op_table(bases[0][order], 0, bases[2][order], 1.0),
                                   ("f64",) if precision == "f64" else ("f64", "f32"))
        # per-dot L panels (a block permutation of every operator's L), FP64 and FP32
        self.lperm = None
        if lperm:
            self._lperm_h = numpy.concatenate(lperm)
            self.lperm = upload(self._lperm_h, dev)
            self._lperm_ops = op_table(L.offsets[order], 0, L.offsets[order], 1.0)
            self._lperm_ops_d = upload(self._lperm_ops, dev)
            self._lperm_span = int(max(len(v[0]) for v in plans.values()))
            self._build_lpan(sparse_w)
        # per-dot R panels (every operator's R blocks permuted), FP64 and FP32
        self.rperm = None
        if rperm:
            self._rperm_h = numpy.concatenate(rperm)
            self.rperm = upload(self._rperm_h, dev)
            rops = op_table(R.offsets[order], 0, R.offsets[order], 1.0)
            self._rperm_ops_d = upload(rops, dev)
            self._rperm_span = int(max(len(v[0]) for v in plans.values()))
            self._build_rpan(sparse_w)
        # L.psi and .R on K-major panels with padded rows (the L panels of a contracted sector,
        # the transposed R panels, the wavefunction's panels): split TF32 on the tcgen05 kernel,
        # and FP64 (on the tensor pipe) or FP32 where the sparse product runs between them
        self.tc1 = self.tc4 = self.d1 = self.d4 = self.f1 = self.f4 = None
        self.direct, self._kmajor = direct, False
        self.lpan64 = self.lpan_f32 = self.lpan_tc = self.rpan64 = self.rpan_f32 = self.rpan_tc = None
        crow = numpy.concatenate(crow_all) if crow_all else numpy.zeros(1, numpy.int64)
        if tc1_classes:
            self._setup_panels1(tc1_classes, order, L, tabs[0], want_tc1, sparse_w)
        if tc4_classes:
            self._setup_panels4(tc4_classes, order, bases[2], R, tabs[3], crow, want_tc4, sparse_w)
        if direct:
            self._build_kmajor()
        # fused W stage (T1 -> T3) and the per-dot two-site MPO blocks it reads
        self.fused = None
        self.wtot = wtot
        if fuse_parts:
            ftab = op_table(bases[0][order], wbase[order], bases[2][order], 1.0)
            self.fused = CompositeStage(fiber_stages(fuse_parts, dev, "sigma23", ftab, fg_budget), "sigma23")
            wst = Stage(wij_parts, dev, "wij", op_table(Wi.offsets[order], Wj.offsets[order], wbase[order], 1.0))
            self.Wij = torch.zeros(max(wtot, 1), dtype=torch.float64, device=dev)
            wst.run(Wi.values, Wj.values, self.Wij, "f64")
            self._Wij32 = None
        # algorithmic bytes per stage (FP64): every operand block read once, output written once
        def stage_bytes(c, t, nop, shared2):
            if len(t) == 0:
                return 0
            u1 = numpy.unique(t[:, 1])
            u2 = numpy.unique(t[:, 2])
            uo = numpy.unique(t[:, 0])
            b1 = c.l1.ndim[u1].sum() * nop
            b2 = c.l2.ndim[u2].sum() * (1 if shared2 else nop)
            bo = c.out.ndim[uo].sum() * nop
            return 8 * (b1 + b2 + bo)

        fb = 0
        for si in range(4 if LOG.enabled else 0):       # only the launch log reads the byte counts
            tot_b = 0
            for key, (ops, *cs, Rl, fused, pan, pan4, fib2, fib3) in sorted(plans.items()):
                if fused is not None and si in (1, 2):
                    continue
                c, t = cs[si]
                tot_b += stage_bytes(c, t, len(ops), si == 0)      # psi is read by every operator
            if self._stages[si] is not None:
                self._stages[si].bytes = float(tot_b)
            if self.wx is not None and si in (1, 2):
                # T1 and the site's MPO in, T3 and the other site's MPO: no T2
                for key, (ops, *cs, Rl, fused, pan, pan4, fib2, fib3) in sorted(plans.items()):
                    (ca, ta), (cb, tb) = cs[1], cs[2]
                    u, wu = (numpy.unique(ta[:, 1]), numpy.unique(ta[:, 2])) if si == 1 else \
                        (numpy.unique(tb[:, 0]), numpy.unique(tb[:, 2]))
                    nb = (ca.l1.ndim[u].sum() + ca.l2.ndim[wu].sum()) if si == 1 else \
                        (cb.out.ndim[u].sum() + cb.l2.ndim[wu].sum())
                    self.wx.bytes += 8.0 * float(nb) * len(ops)
        for key, (ops, *cs, Rl, fused, pan, pan4, fib2, fib3) in sorted(plans.items()):
            if fused is not None and LOG.enabled:
                fb += stage_bytes(fused[1], fused[2], len(ops), False)
        if self.fused is not None:
            self.fused.bytes = float(fb)
        for st, ref in ((self.tc1, 0), (self.d1, 0), (self.f1, 0), (self.tc4, 3), (self.d4, 3), (self.f4, 3)):
            if st is not None:
                st.bytes = self._stages[ref].bytes
        # FLOPs of the reference's four-contraction chain (tensordotCAL pair GEMMs),
        # whatever the fusion used here
        self.flops = 0.0
        for key, (ops, *cs, Rl, fused, pan, pan4, fib2, fib3) in sorted(plans.items()):
            for si, (c, t) in enumerate(cs):
                fl = pair_flops(c, t) * len(ops)
                self.flops += fl
                if self.wx is not None and si in (1, 2):
                    self.wx.flops += fl
        self.ndim0 = psi_layout.size
        # W panels of the dense fiber-group stages, gathered now (per dot) rather than in
        # the first matrix-vector product
        if torch.device(dev).type == "cuda":
            s = torch.cuda.current_stream(dev).cuda_stream
            wsets = [(self._stages[1], self.Wi), (self._stages[2], self.Wj)]
            for st, wset in wsets if self.wx is None else []:
                for sub in (st.subs if isinstance(st, CompositeStage) else [st]):
                    if isinstance(sub, FiberStage) and sub.ntasks and sub.fgemm:
                        sub.wpanel(wset.values, s)
                        if precision != "f64":
                            sub.wpanel(wset.f32(), s)

    def _chain(self, Ll, W1, W2, Rl, use_fiber, panel1, panel4, r_fast=False):
        """The four contractions of one operator class with their block pairs, and the panel
        forms of the first and the last one (None where a class has none)."""
        ax, _, _, live, _ = self._fiber_args
        c1 = Contraction(Ll, self.psi, ax[0])
        t1 = c1.triples if live is None else prune(c1.triples, live2=live)
        # L.psi as dense panel GEMMs (T1 blocks stored panel by panel)
        pan = panel_sigma1(Ll, self.psi, t1, c1.out.nblks) if panel1 else None
        c2 = Contraction(c1.out, W1, ax[1])
        t2 = prune(c2.triples, live1=live_blocks(c1.out, t1))
        c3 = Contraction(c2.out, W2, ax[2])
        t3 = prune(c3.triples, live1=live_blocks(c2.out, t2))
        c4 = Contraction(c3.out, Rl, ax[3])
        t4 = c4.triples if live is None else c4.triples[live[c4.triples[:, 0]]]
        # .R as dense panel GEMMs (T3 blocks written into sigma-block panels, R blocks
        # permuted into per-sector panels once per dot)
        pan4 = panel_sigma4(c3.out, Rl, self.psi, t4, r_fast) if (use_fiber and panel4) else None
        return (c1, t1), (c2, t2), (c3, t3), (c4, t4), pan, pan4

    @staticmethod
    def _fiber_pair(c1, c2, t2, c3, t3, t1off, o3):
        """.W_i and .W_{i+1} on the fiber kernel: T2 stored column by column (its physical
        axes have extent 1, so a T2 block's columns are the next contraction's rows and its
        fibers that contraction's fibers), read back with contiguous fibers."""
        cm = bool(unit_phys_t2(c2.out))
        fib2 = compile_fiber(c2, t2, 0, 0, in_off=t1off, out_colmajor=cm)
        cm = cm and fib2 is not None
        fib3 = compile_fiber(c3, t3, 3, 0 if cm else 1, **o3)
        if fib3 is None and cm and not o3:
            fib2 = compile_fiber(c2, t2, 0, 0, in_off=t1off)       # T2 packed for the grouped GEMM
        return fib2, fib3

    @property
    def stages(self):
        """The four contractions as separate stages.  With the sparse product the two
        MPO-site ones are not part of a matrix-vector product; they are compiled when asked
        for (lockstep batches run the stages of many operators in common launches)."""
        if self.wx is not None and self._stages[1] is None:
            ax, groups, qkey, live, fg_budget = self._fiber_args
            fib = [[], []]
            pos = 0
            for key, ops in sorted(groups.items()):
                rng = (pos, pos + len(ops))
                pos += len(ops)
                i0 = ops[0]
                (c1, _), (c2, t2), (c3, t3), _, pan, pan4 = self._chain(
                    self._lays[0][i0], self.Wi.layouts[i0], self.Wj.layouts[i0], flip_right(self._lays[1][i0], qkey),
                    True, True, True, True)
                f2, f3 = self._fiber_pair(c1, c2, t2, c3, t3, pan["t1off"],
                                          {"out_off": pan4["t3off"], "out_fhs": pan4["t3fhs"],
                                           "out_flo": pan4["t3flo"], "extra_out": pan4["needed"],
                                           "out_rfast": True})
                if f2 is None or f3 is None:
                    raise RuntimeError("fiber groups of a sparse two-site plan could not be compiled")
                fib[0].append(f2 + (rng,))
                fib[1].append(f3 + (rng,))
            for k in (0, 1):
                name = "sigma%d" % (k + 2)
                self._stages[k + 1] = CompositeStage(
                    fiber_stages(fib[k], self.ws.device, name, self._tabs[k + 1], fg_budget), name)
        return self._stages

    def rebind(self, L, R):
        """Use new environment values with the same block layouts (cached plan)."""
        if (len(L.layouts) != len(self._lays[0]) or len(R.layouts) != len(self._lays[1])
                or any(a is not b for a, b in zip(L.layouts, self._lays[0]))
                or any(a is not b for a, b in zip(R.layouts, self._lays[1]))):
            raise ValueError("rebind: environment layouts differ from the compiled plan")
        self.L, self.R = L, R
        if self.lperm is not None:
            self._build_lpan(self.d1 is not None)
        if self.rperm is not None:
            self._build_rpan(self.d4 is not None)
        self._kmajor = False
        if self.direct:
            self._build_kmajor()

    def _setup_panels4(self, tc4_classes, order, t3bases, R, st4_ops, crow, tc, f64):
        from .engine import TCPanelStage, tc_sigma4_units
        dev = self.ws.device
        classes, t3b, rtb, rts, descs = [], [], [], [], []
        rt_tot = 0
        flops = 0.0
        for (rng, pan4, crow_n) in tc4_classes:
            sec = dict(pan4["sectors"])
            sec["crow_base"] = sec["crow_base"] + crow_n
            ops_c = order[rng[0]:rng[1]]
            t3stride = int(t3bases[ops_c[1]] - t3bases[ops_c[0]]) if len(ops_c) > 1 else \
                (int(pan4["t3size"]) + 31) // 32 * 32
            opstride = (int(pan4["rtsize"]) + 31) // 32 * 32
            classes.append((list(range(rng[0], rng[1])), sec, t3stride))
            t3b.append(int(t3bases[ops_c[0]]))
            rtb.append(rt_tot)
            rts.append(opstride)
            src, dst, dU, st3 = pan4["rperm_t"]
            d = numpy.zeros(len(src), BPERM_DT)
            d["src_off"], d["dst_off"] = src, dst
            d["d0"], d["d1"], d["d2"] = dU[:, 0], dU[:, 1], dU[:, 2]
            d["s0"], d["s1"], d["s2"] = st3
            d["op_b"], d["op_e"] = rng
            descs.append(d)
            rt_tot += opstride * len(ops_c)
            flops += 2.0 * float((sec["M"] * sec["N"] * sec["K"]).sum()) * len(ops_c)
        rt_tot = (rt_tot + 31) // 32 * 32
        if tc:
            units, maps = tc_sigma4_units(classes, None, t3b, rtb, rts, rt_tot)
            self.tc4 = TCPanelStage("sigma4", units, maps, st4_ops, crow, flops, dev)
        # .R writes every element of every partial vector (none twice)
        self._part_full = sum(len(poss) for poss, _, _ in classes) == len(order) and \
            all(int((sec["M"] * sec["N"]).sum()) == self.psi.size for _, sec, _ in classes)
        self._rt_total = rt_tot
        self._rt_descs = numpy.concatenate(descs)
        self._rt_descs_d = upload(self._rt_descs, dev)
        base = numpy.zeros(len(order), dtype=numpy.int64)
        for (poss, sec, _), b0, st in zip(classes, rtb, rts):
            base[poss] = b0 + st * numpy.arange(len(poss))
        self._rt_ops_d = upload(op_table(R.offsets[order], 0, base, 1.0), dev)
        self._rt_span = int(max(len(c[0]) for c in classes))
        if f64:
            ops = st4_ops.copy()
            ops["b_base"] = base
            for kind in ("f64", "f32") if self.precision == "f32" else ("f64",):
                parts = [(dpanel_units(sec["M"], sec["N"], sec["K"], sec["Kp"], sec["Kp"], sec["t3pan"],
                                       sec["rtoff"], sec["crow_base"], "row", kind=kind), (poss[0], poss[-1] + 1))
                         for (poss, sec, _) in classes]
                st = DPanelStage("sigma4", parts, ops, dev, flops, crow=crow, longest_first=True, kind=kind)
                self.d4, self.f4 = (st, self.f4) if kind == "f64" else (self.d4, st)

    def _setup_panels1(self, tc1_classes, order, L, st1_ops, tc, f64):
        from .engine import TCPanelStage, tc_sigma1_units
        dev = self.ws.device
        live = numpy.unique(numpy.concatenate([t["blocks"] for _, t in tc1_classes]))
        gidx, info, cols = psi_panels(self.psi, live)
        self._psi_total = (len(gidx) + 31) // 32 * 32
        self._psi_gidx = torch.from_numpy(numpy.concatenate(
            [gidx, numpy.full(self._psi_total - len(gidx), -1, dtype=numpy.int64)])).to(dev)
        classes, lpb, lps, descs = [], [], [], []
        tot = 0
        base = numpy.zeros(len(order), dtype=numpy.int64)
        for (rng, tcd) in tc1_classes:
            poss = list(range(rng[0], rng[1]))
            stride = (int(tcd["lpsize"]) + 31) // 32 * 32
            classes.append((poss, tcd))
            lpb.append(tot)
            lps.append(stride)
            base[poss] = tot + stride * numpy.arange(len(poss))
            src, dst, dL, kp = tcd["lperm_t"]
            d = numpy.zeros(len(src), BPERM_DT)
            d["src_off"], d["dst_off"] = src, dst
            d["d0"], d["d1"], d["d2"] = dL[:, 0], dL[:, 1], dL[:, 2]
            d["s0"], d["s1"], d["s2"] = dL[:, 1] * kp, kp, 1
            d["op_b"], d["op_e"] = rng
            descs.append(d)
            tot += stride * len(poss)
        self._lp_total = (tot + 31) // 32 * 32
        if tc:
            units, maps, segs = tc_sigma1_units(classes, info, cols, lpb, lps, self._lp_total, self._psi_total)
            self.tc1 = TCPanelStage("sigma1", units, maps, st1_ops, None, self._stages[0].flops, dev, segs=segs)
        if f64:
            ops = st1_ops.copy()
            ops["a_base"], ops["b_base"] = base, 0
            for kind in ("f64", "f32") if self.precision == "f32" else ("f64",):
                parts, tab = self._dpanel1_units(classes, info, cols, kind)
                st = DPanelStage("sigma1", parts, ops, dev, self._stages[0].flops, cols=tab, kind=kind)
                self.d1, self.f1 = (st, self.f1) if kind == "f64" else (self.d1, st)
        self._lp_descs = numpy.concatenate(descs)
        self._lp_descs_d = upload(self._lp_descs, dev)
        self._lp_ops_d = upload(op_table(L.offsets[order], 0, base, 1.0), dev)
        self._lp_span = int(max(len(c[0]) for c in classes))

    @staticmethod
    def _dpanel1_units(classes, info, cols, kind):
        """Units and column table of L.psi: the psi panel of a contracted sector times
        the class's L panel of that sector; column c of psi block j of sector l' is column c of
        the T1 panel at t1pan_j (rows N_j apart)."""
        secs = sorted(info)
        col0 = dict(zip(secs, (numpy.cumsum([info[s][1] for s in secs]) - [info[s][1] for s in secs]).tolist()))
        ncol = int(sum(info[s][1] for s in secs))
        parts, tabs = [], []
        for poss, tc in classes:
            base = ncol * len(tabs)
            tab = numpy.zeros(max(ncol, 1), DCOL_DT)
            tab["off"] = -1
            nj, pan = numpy.asarray(tc["Nj"], dtype=numpy.int64), numpy.asarray(tc["t1pan"], dtype=numpy.int64)
            at = numpy.array([col0[cols[b][0]] + cols[b][1] for b in tc["blocks"].tolist()], dtype=numpy.int64)
            own = numpy.repeat(numpy.arange(len(nj)), nj)
            loc = numpy.arange(int(nj.sum())) - numpy.repeat(numpy.cumsum(nj) - nj, nj)
            if len(pan) and int(pan.max()) + int(nj.max()) >= 2 ** 31:
                raise ValueError("T1 panel offsets exceed the column record")
            tab["off"][at[own] + loc] = pan[own] + loc
            tab["ld"][at[own] + loc] = nj[own]
            tabs.append(tab)
            sec = [int(s) for s in tc["sectors"]]
            N = [info[s][1] for s in sec]
            u = dpanel_units(tc["M"], N, tc["K"], tc["Kp"], [info[s][3] for s in sec], tc["lpoff"],
                             [info[s][0] for s in sec], [base + col0[s] for s in sec], "col", kind=kind)
            parts.append((u, (poss[0], poss[-1] + 1)))
        return parts, numpy.concatenate(tabs)

    def _build_kmajor(self):
        if self.tc4 is not None or self.d4 is not None:
            self._build_rpan_k()
        if self.tc1 is not None or self.d1 is not None:
            self._build_lpan_k()
        # (made by every replay where a graph is captured)
        self._kmajor = torch.device(self.ws.device).type != "cuda" or not torch.cuda.is_current_stream_capturing()

    def _build_lpan_k(self):
        """K-major L panels [M x Kp] per sector: FP32 hi plane then lo plane for the tcgen05 kernel,
        FP64 and FP32 for the others."""
        n = self._lp_total
        if self.f1 is not None:
            self.lpan_f32 = torch.empty(max(n, 1), dtype=torch.float32, device=self.ws.device)
            block_permute(self._lp_descs_d, len(self._lp_descs), self._lp_span, self._lp_ops_d, self.L.values,
                          self.lpan_f32)
        if self.d1 is not None:
            self.lpan64 = torch.empty(max(n, 1), dtype=torch.float64, device=self.ws.device)
            block_permute(self._lp_descs_d, len(self._lp_descs), self._lp_span, self._lp_ops_d, self.L.values,
                          self.lpan64)
        if self.tc1 is None:
            return
        self.lpan_tc = torch.zeros(2 * max(n, 1), dtype=torch.float32, device=self.ws.device)
        block_permute(self._lp_descs_d, len(self._lp_descs), self._lp_span, self._lp_ops_d, self.L.values,
                      self.lpan_tc)
        tf32_split(self.lpan_tc[:n], self.lpan_tc[n:2 * n])

    def _build_rpan_k(self):
        """K-major R panels [D_r' x Kp] per sector: FP32 hi plane then lo plane for the tcgen05
        kernel, FP64 and FP32 for the others."""
        n = self._rt_total
        if self.f4 is not None:
            self.rpan_f32 = torch.empty(max(n, 1), dtype=torch.float32, device=self.ws.device)
            block_permute(self._rt_descs_d, len(self._rt_descs), self._rt_span, self._rt_ops_d, self.R.values,
                          self.rpan_f32)
        if self.d4 is not None:
            self.rpan64 = torch.empty(max(n, 1), dtype=torch.float64, device=self.ws.device)
            block_permute(self._rt_descs_d, len(self._rt_descs), self._rt_span, self._rt_ops_d, self.R.values,
                          self.rpan64)
        if self.tc4 is None:
            return
        self.rpan_tc = torch.zeros(2 * max(n, 1), dtype=torch.float32, device=self.ws.device)
        block_permute(self._rt_descs_d, len(self._rt_descs), self._rt_span, self._rt_ops_d, self.R.values,
                      self.rpan_tc)
        tf32_split(self.rpan_tc[:n], self.rpan_tc[n:2 * n])

    def _build_rpan(self, later=False):
        """Panels of the separate .R stage; later: made when that stage asks for them."""
        self.Rpan = self._Rpan32 = None
        if not later:
            self.Rpan = torch.empty(max(self.R.total, 1), dtype=torch.float64, device=self.ws.device)
            block_permute(self.rperm, len(self._rperm_h), self._rperm_span, self._rperm_ops_d, self.R.values,
                          self.Rpan)

    def b4(self, kind):
        """Second operand of the .R contraction (R panels, or R itself without panels)."""
        if self.rperm is not None:
            if kind == "f64":
                if self.Rpan is None:
                    self._build_rpan()
                return self.Rpan
            if self._Rpan32 is None:
                self._Rpan32 = torch.empty(max(self.R.total, 1), dtype=torch.float32, device=self.ws.device)
                block_permute(self.rperm, len(self._rperm_h), self._rperm_span, self._rperm_ops_d,
                              self.R.values, self._Rpan32)
            return self._Rpan32
        return self.R.values if kind == "f64" else self.R.f32()

    def _build_lpan(self, later=False):
        """Panels of the separate L.psi stage; later: made when that stage asks for them."""
        self.Lpan = self._Lpan32 = None
        if not later:
            self.Lpan = torch.empty(max(self.L.total, 1), dtype=torch.float64, device=self.ws.device)
            block_permute(self.lperm, len(self._lperm_h), self._lperm_span, self._lperm_ops_d, self.L.values,
                          self.Lpan)

    def lpan32(self):
        if self._Lpan32 is None:
            self._Lpan32 = torch.empty(max(self.L.total, 1), dtype=torch.float32, device=self.ws.device)
            block_permute(self.lperm, len(self._lperm_h), self._lperm_span, self._lperm_ops_d, self.L.values,
                          self._Lpan32)
        return self._Lpan32

    def a1(self, kind):
        """First operand of the L.psi contraction (L panels, or L itself without panels)."""
        if self.lperm is not None:
            if kind == "f64" and self.Lpan is None:
                self._build_lpan()
            return self.Lpan if kind == "f64" else self.lpan32()
        return self.L.values if kind == "f64" else self.L.f32()

    def release(self):
        """Drop the references to the environment values (the plan stays valid)."""
        self.L = self.R = None
        self.Lpan = self._Lpan32 = None
        self.Rpan = self._Rpan32 = None
        self.rpan_tc = self.rpan64 = self.rpan_f32 = None
        self.lpan_tc = self.lpan64 = self.lpan_f32 = None

    def wij32(self):
        if self._Wij32 is None:
            self._Wij32 = self.Wij.to(torch.float32)
        return self._Wij32

    def scratch_bytes(self):
        return 8 * sum(self.tot)

    def check_device_status(self):
        """Raise if a tensor-core launch of this plan gave up a bounded wait (its device
        error flag, qc_tcpanel_status): its output would be incomplete.  Reads one int."""
        if (self.tc1 is not None or self.tc4 is not None) and torch.device(self.ws.device).type == "cuda":
            st = native.lib().qc_tcpanel_status(1)
            if st != 0:
                raise RuntimeError("tensor-core panel kernel: a bounded wait expired (status %d); the sigma of "
                                   "this dot is incomplete" % st)

    def work_groups(self):
        """The plan's device work-item groups in stage order, as the C-ABI's
        qc_sigma_f64_noalloc takes them: (stage, kind, tasks, ntasks, opspan, contribs,
        tile_cfg), kind one of native.GROUP_BGEMM / GROUP_PANEL / GROUP_FIBER.  Groups
        that read the per-dot panels (the tensor-core tiles of a panel stage included)
        are GROUP_PANEL; the fused two-site W stage counts as a fiber group of stage 1."""
        out = []

        def walk(st, si, kind=None):
            if st is None:
                return
            if isinstance(st, CompositeStage):
                for x in st.subs:
                    walk(x, si, kind)
            elif isinstance(st, PanelStage):
                for (cfg, tk, dt, span) in st.groups:
                    out.append((si, native.GROUP_PANEL, dt.data_ptr(), len(tk), span, 0, cfg))
                walk(st.tc, si, native.GROUP_PANEL)
            elif isinstance(st, FiberStage):
                if st.ntasks:
                    out.append((si, native.GROUP_FIBER, st.d[0].data_ptr(), st.ntasks, st.span, 0, 0))
            else:
                for (cfg, tk, ct, dt, dc, span) in st.groups:
                    out.append((si, kind or native.GROUP_BGEMM, dt.data_ptr(), len(tk), span, dc.data_ptr(), cfg))

        for si, st in enumerate(self.stages):
            walk(st, si)
            if si == 1:
                walk(self.fused, 1, native.GROUP_FIBER)
            if si == 3 and self.tc4 is not None:
                out.append((3, native.GROUP_PANEL, self.tc4.d_units.data_ptr(), self.tc4.ntasks, 1, 0, 0))
            if si == 0 and self.tc1 is not None:
                out.append((0, native.GROUP_PANEL, self.tc1.d_units.data_ptr(), self.tc1.ntasks, 1, 0, 0))
        return out

    def _native_plan(self, kind):
        """The launches of one product in `kind` as a native.SigmaPlan: pointers to device tables
        that this operator owns."""
        p = self._plans.get(kind)
        if p is None:
            d, w = self.wx.d, self.wx
            first, last = {"f64": (self.d1, self.d4), "f32": (self.f1, self.f4), "tf32x3": (self.tc1, self.tc4)}[kind]
            p = native.SigmaPlan(("f64", "f32", "tf32x3").index(kind), self.nops, int(not self._part_full), 0, self.ndim0,
                                 self._psi_gidx.numel(), self._psi_gidx.data_ptr(), first.record(), last.record())
            n = 0
            if w.ntasks:
                p.deltas, p.groups, p.rows, p.dops, p.octs, p.ent_r, p.wops = (
                    d[k].data_ptr() for k in ("deltas", "groups", "rows", "dops", "octs", "ent_r", "ops"))
                wk = "f64" if kind == "f64" else "f32"
                p.ent_w = w.weights(wk).data_ptr()
                for tile, host, dev, maxr, maxo in w.items(wk):
                    p.tiles[n] = native.SigmaTiles(dev.data_ptr(), len(host), tile, maxr, maxo, 0)
                    n += 1
            self._plans[kind] = p = (ctypes.byref(p), p, n + 4)
        return p

    def _run_panels(self, kind, x, y):
        dt = torch.float64 if kind == "f64" else torch.float32
        ws = self.ws
        ref, _, launches = self._native_plan(kind)
        psi = ws.get("psi_pan", self._psi_total * (2 if kind == "tf32x3" else 1), dt)
        t3 = ws.get("t3", self.tot[2], dt)
        if kind == "tf32x3":
            lpan, rpan = self.tc1.maps(self.lpan_tc, psi), self.tc4.maps(t3, self.rpan_tc)
        else:
            lpan, rpan = (self.lpan64, self.rpan64) if kind == "f64" else (self.lpan_f32, self.rpan_f32)
        check(native.lib().qc_sigma_panels(
            ref, lpan.data_ptr(), rpan.data_ptr(), x.data_ptr(), psi.data_ptr(),
            ws.get("t1", self.tot[0], dt).data_ptr(), t3.data_ptr(),
            ws.get("part", self.nops * self.ndim0, dt).data_ptr(), y.data_ptr(), _stream(y.device)),
            "qc_sigma_panels")
        LOG.launches += launches
        return y

    def _x32(self, x):
        x32 = self.ws.get("x32", self.ndim0, torch.float32)
        convert(x, x32)
        return x32

    def __call__(self, x, y=None, precision=None):
        """x: device tensor (ndim0,) float64 -> y = H x (float64).

        precision overrides the operator's precision for this call ("f64" runs the
        same plan, tensor-core tiles included, on the FP64 engine)."""
        ws = self.ws
        prec = precision or self.precision
        if y is None:
            y = torch.empty(self.ndim0, dtype=torch.float64, device=ws.device)
        if not self._kmajor:
            self._build_kmajor()
        # in panel form all through: one native call (the launch log times the stages one by one)
        if self.wx is not None and x.is_cuda and not LOG.enabled and (
                prec == "f64" or (prec == "f32" and self.f1 is not None) or
                (prec == "tf32x3" and self.tc1 is not None and self.tc4 is not None and self._s0_generic is None)):
            return self._run_panels(prec, x, y)
        if prec == "f64":
            T1 = ws.get("t1", self.tot[0], torch.float64)
            T3 = ws.get("t3", self.tot[2], torch.float64)
            P = ws.get("part", self.nops * self.ndim0, torch.float64)
            s = self._stages
            if self.wx is not None:
                pt = ws.get("psi_pan", self._psi_total, torch.float64)
                gather_pad(x, self._psi_gidx, pt)
                self.d1.run(self.lpan64, pt, T1)
                self.wx.run(T1, None, T3, "f64")
                if not self._part_full:
                    P[:self.nops * self.ndim0].zero_()
                self.d4.run(T3, self.rpan64, P)
                return reduce_ops(P, self.nops, self.ndim0, y)
            else:
                s[0].run(self.a1("f64"), x, T1, "f64")
                T2 = ws.get("t2", self.tot[1], torch.float64)
                s[1].run(T1, self.Wi.values, T2, "f64")
                s[2].run(T2, self.Wj.values, T3, "f64")
            if self.fused is not None:
                self.fused.run(T1, self.Wij, T3, "f64")
            P[:self.nops * self.ndim0].zero_()
            s[3].run(T3, self.b4("f64"), P, "f64")
            return reduce_ops(P, self.nops, self.ndim0, y)
        kind = prec if prec in ("tf32", "tf32x3") else "f32"
        T1 = ws.get("t1", self.tot[0], torch.float32)
        T3 = ws.get("t3", self.tot[2], torch.float32)
        y32 = ws.get("y32", self.ndim0, torch.float32)
        P = ws.get("part", self.nops * self.ndim0, torch.float32)
        s = self._stages
        if self.tc1 is not None and kind == "tf32x3":
            pt = ws.get("psiT", 2 * self._psi_total, torch.float32)
            gather_split(x, self._psi_gidx, pt[:self._psi_total], pt[self._psi_total:2 * self._psi_total])
            self.tc1.run(self.lpan_tc, pt, T1)
            if self._s0_generic is not None:
                self._s0_generic.run(self.a1("f32"), self._x32(x), T1, "f32")
        elif self.f1 is not None and kind == "f32":
            pt = ws.get("psi_pan", self._psi_total, torch.float32)
            gather_pad(x, self._psi_gidx, pt)
            self.f1.run(self.lpan_f32, pt, T1)
        else:
            s[0].run(self.a1("f32"), self._x32(x), T1, kind)
        if self.wx is not None:
            self.wx.run(T1, None, T3, "f32")
        else:
            T2 = ws.get("t2", self.tot[1], torch.float32)
            s[1].run(T1, self.Wi.f32(), T2, "f32")
            s[2].run(T2, self.Wj.f32(), T3, "f32")
        if self.fused is not None:
            self.fused.run(T1, self.wij32(), T3, "f32")
        P[:self.nops * self.ndim0].zero_()
        if self.tc4 is not None and kind == "tf32x3":
            self.tc4.run(T3, self.rpan_tc, P)
        elif self.f4 is not None and kind == "f32":
            self.f4.run(T3, self.rpan_f32, P)
        else:
            s[3].run(T3, self.b4("f32"), P, kind)
        reduce_ops(P, self.nops, self.ndim0, y32)
        convert(y32, y)
        return y


_DENSE_STAGES = {}
PANEL_OPS = 65535         # operators of one panel task: the launch's second grid extent


def _diag_stages(dev, nops, A, Ab, Ac, ldim, rdim, hp):
    """The three dense stages of the diagonal; they depend only on the dimensions (and the
    operator weights), so dots of equal shape share one set of device work lists."""
    key = (str(dev), nops, A, Ab, Ac, ldim, rdim, hp.tobytes())
    hit = _DENSE_STAGES.get(key)
    if hit is not None:
        return hit
    p = numpy.repeat(numpy.arange(nops), 16)
    nm = numpy.tile(numpy.arange(16), nops)
    n, m = nm // 4, nm % 4

    def stage(name, M, N, K, ops, count, crow=None, lda=None):
        z = numpy.zeros(1, dtype=numpy.int64)
        g = (z, z, z, z + M, z + N, z + K, z if crow is not None else z - 1, z + (K if lda is None else lda))
        parts = {}
        for b in range(0, count, PANEL_OPS):        # (spin projection: 16 x operators x quadrature points)
            for c, t in compile_panels(g, (b, min(b + PANEL_OPS, count))).items():
                parts.setdefault(c, []).append(t)
        return PanelStage(parts, dev, name, ops, crow=crow)

    # X[p, n, m][a, c] = sum_b W1[p, n][a, b] W2[p, m][b, c]
    sX = stage("diagX", A, Ac, Ab, op_table((p * 4 + n) * A * Ab, (p * 4 + m) * Ab * Ac, (p * 16 + nm) * A * Ac, 1.0),
               16 * nops)
    # T[nm][l, (p, c)] = w_p sum_a Ld[p][l, a] X[p, nm][a, c]
    sT = stage("diagT", ldim, Ac, A, op_table(p * ldim * A, (p * 16 + nm) * A * Ac, nm * ldim * nops * Ac + p * Ac,
                                              hp[p]), 16 * nops, crow=numpy.arange(ldim, dtype=numpy.int64) * nops * Ac)
    # D[nm][l, r] = sum_(p, c) T[nm][l, (p, c)] Rd[(p, c), r]
    k = numpy.arange(16)
    sD = stage("diagD", ldim, rdim, nops * Ac, op_table(k * ldim * nops * Ac, 0, k * ldim * rdim, 1.0), 16)
    out = (sX, sT, sD)
    if len(_DENSE_STAGES) > 256:
        _DENSE_STAGES.clear()
    _DENSE_STAGES[key] = out
    return out


_DIAG_CACHE = {}


def _cached(key, lay, build):
    hit = _DIAG_CACHE.get(key)
    if hit is not None and hit[0] is lay:
        return hit[1]
    if len(_DIAG_CACHE) > 4096:
        _DIAG_CACHE.clear()
    val = build()
    _DIAG_CACHE[key] = (lay, val)
    return val


def _ragged(n):
    """Block id and in-block position of every element of blocks with n elements each."""
    n = numpy.asarray(n, dtype=numpy.int64)
    b = numpy.repeat(numpy.arange(len(n)), n)
    e = numpy.arange(int(n.sum()), dtype=numpy.int64) - numpy.repeat(numpy.cumsum(n) - n, n)
    return b, e


def _neutral(lay, axis):
    """First neutral state of every sector of an MPO bond among those of quantum number zero (-1:
    another quantum number), and the number of neutral states.  Diagonal blocks E[a, l, l] and
    W[a, b, n, n] between them are all that the diagonal of H_eff reads."""
    z = (numpy.rint(2 * numpy.asarray(lay.qsyms[axis])) == 0).all(axis=1)
    n = numpy.where(z, numpy.asarray(lay.ndims[axis], dtype=numpy.int64), 0)
    return numpy.where(z, numpy.cumsum(n) - n, -1), int(n.sum())


def _env_diag_map(lay, A, ncol, kfast):
    """Environment E[a, l, l], a neutral -> a dense [ncol x A] (kfast) or [A x ncol] matrix:
    source index of every dense element, -1 for none."""
    def build():
        idx = lay.idx_allowed
        sa, s1, s2 = numpy.unravel_index(idx, tuple(lay.nsyms))
        a0 = _neutral(lay, 0)[0][sa]
        keep = (s1 == s2) & (a0 >= 0)
        idx, s1, a0 = idx[keep], s1[keep], a0[keep]
        d = lay.block_dims(idx) if len(idx) else numpy.zeros((0, 3), dtype=numpy.int64)
        da, dl = d[:, 0], d[:, 1]
        b, e = _ragged(da * dl)
        w, u = e // dl[b], e % dl[b]
        src = lay.ioff[idx][b] + w * dl[b] * dl[b] + u * dl[b] + u
        w = w + a0[b]
        col = lay.secoff[1][s1][b] + u
        out = numpy.full(A * ncol, -1, dtype=numpy.int64)
        out[col * A + w if kfast else w * ncol + col] = src
        return out
    return _cached(("e", id(lay), A, ncol, kfast), lay, build)


def _w_diag_map(lay, A, B):
    """MPO site operator W[a, b, n, n], a and b neutral -> a dense [4 x A x B] array."""
    def build():
        idx = lay.idx_allowed
        sa, sb, n, n_ = numpy.unravel_index(idx, tuple(lay.nsyms))
        a0, b0 = _neutral(lay, 0)[0][sa], _neutral(lay, 1)[0][sb]
        keep = (n == n_) & (a0 >= 0) & (b0 >= 0)
        idx, n, a0, b0 = idx[keep], n[keep], a0[keep], b0[keep]
        d = lay.block_dims(idx) if len(idx) else numpy.zeros((0, 4), dtype=numpy.int64)
        da, db = d[:, 0], d[:, 1]
        b, e = _ragged(da * db)
        w, v = e // db[b], e % db[b]
        out = numpy.full(4 * A * B, -1, dtype=numpy.int64)
        out[(n[b] * A + a0[b] + w) * B + b0[b] + v] = lay.ioff[idx][b] + w * db[b] + v
        return out
    return _cached(("w", id(lay), A, B), lay, build)


def _psi_diag_gather(ql, ldim, rdim):
    """Packed wavefunction position -> index of the dense [16, ldim, rdim] diagonal
    (qc_psi_diag_gather, host code of the native library)."""
    def build():
        blocks = numpy.ascontiguousarray(ql.idx_allowed, dtype=numpy.int64)
        gat = numpy.empty(max(ql.size, 1), dtype=numpy.int64)
        check(native.lib().qc_psi_diag_gather(len(blocks), native.ptr(blocks), native.ptr(ql.nsyms),
                                              native.ptr(ql.ndims_cat), native.ptr(ql.ioff), ldim, rdim, ql.size,
                                              native.ptr(gat)), "qc_psi_diag_gather")
        return gat[:ql.size]
    return _cached(("p", id(ql), ldim, rdim), ql, build)


class DiagOperator(object):
    """Davidson diagonal in the packed wavefunction layout (HDiagQt, two-site).

    Only the neutral sector of the MPO bonds enters (13 of 98 states at K=24): three dense
    panel GEMMs on FP64 tensor products over it, all operators in the contracted extent of the
    last one.  K=24, D=300, host result included: 3.03 -> 0.32 ms (218 us on the device, 131
    of them the last product; the whole bond took 2.8 ms)."""

    def __init__(self, ws, isite, psi_layout, L, R, Wi, Wj, qkey, opers, hpwts):
        dev = ws.device
        self.ws = ws
        nops = len(opers)
        ql = psi_layout
        ldim = int(ql.shape[0])
        rdim = int(ql.shape[3])
        # extents of the neutral MPO bond sectors (the largest over the operators, zero-padded)
        A = max(1, max(_neutral(l, 0)[1] for l in L.layouts))
        Ab = max(1, max(_neutral(l, 1)[1] for l in Wi.layouts))
        Ac = max(1, max(_neutral(l, 0)[1] for l in R.layouts))
        self.dims = (A, Ab, Ac, ldim, rdim)
        # ---- source of every element of the dense operands (host; cached per interned layout)
        def cat(tset, build):
            m = [build(tset.layouts[i]) for i in range(nops)]
            return torch.from_numpy(numpy.concatenate([numpy.where(x >= 0, x + o, -1)
                                                       for x, o in zip(m, tset.offsets)])).to(dev)

        self.maps = [(cat(L, lambda l: _env_diag_map(l, A, ldim, True)), "ld", L),
                     (cat(R, lambda l: _env_diag_map(l, Ac, rdim, False)), "rd", R),
                     (cat(Wi, lambda l: _w_diag_map(l, A, Ab)), "w1", Wi),
                     (cat(Wj, lambda l: _w_diag_map(l, Ab, Ac)), "w2", Wj)]
        # ---- packed output gather: psi block (sl, n, m, sr), element (u, v) ----
        gat = _psi_diag_gather(ql, ldim, rdim)
        self.gather = torch.from_numpy(gat).to(dev)
        self.ndim0 = ql.size
        # ---- three dense GEMM stages (shared by dots of equal dimensions) ----
        hp = numpy.asarray(hpwts, dtype=numpy.float64)
        self.sX, self.sT, self.sD = _diag_stages(dev, nops, A, Ab, Ac, ldim, rdim, hp)
        self.nX = nops * 16 * A * Ac
        self.nT = nops * 16 * Ac * ldim
        self.nD = 16 * ldim * rdim
        self.flops = self.sX.flops + self.sT.flops + self.sD.flops

    def rebind(self, L, R):
        """Use new environment values with the same block layouts (cached plan)."""
        sub = {"ld": L, "rd": R}
        self.maps = [(idx, name, sub[name] if name in sub else tset) for (idx, name, tset) in self.maps]

    def release(self):
        self.rebind(None, None)

    def __call__(self):
        ws = self.ws
        bufs = {}
        for (idx, name, tset) in self.maps:
            bufs[name] = gather_pad(tset.values, idx, ws.get("diag_" + name, idx.numel(), torch.float64))
        X = ws.get("diag_x", self.nX, torch.float64)
        T = ws.get("diag_t", self.nT, torch.float64)
        D = ws.get("diag_d", self.nD, torch.float64)
        self.sX.run(bufs["w1"], bufs["w2"], X, "f64")
        self.sT.run(bufs["ld"], X, T, "f64")
        self.sD.run(T, bufs["rd"], D, "f64")
        out = torch.empty(self.ndim0, dtype=torch.float64, device=ws.device)
        return gather(D, self.gather, out)


class Renormalizer(object):
    """New environments of every operator after a decimation (renormQt_H00).

    status 'L': L'[b, r, r'] = sum site*[l, n, r] L[a, l, l'] W[a, b, n, n'] site[l', n', r']
    status 'R': the mirror image with W's bond indices flipped (kernelQt.py:723-740).

    With x, y the bra and ket states of the old bond, z, z' those of the new one and S the
    site tensor, three stages over all operators: T1[a, x, n, z'] = E[a, x, y] S[y, n, z']
    (panel GEMM), T2[b, x, n', z'] = W T1 (the sparse MPO stage, fibers (x, z')), and
    E'[b, z, z'] = S*[(x, n'), z] T2[(x, n'), (b, z')] (panel GEMM, T2 as [K x M]).  Dots whose
    blocks have no such form run three grouped block GEMMs.
    """

    def __init__(self, ws, isite, status, site_layout, E, W, opers, panels=None):
        """panels: the panel form (None: on a GPU, where the blocks allow it)."""
        self.ws, self.status = ws, status
        self._args = (ws, isite, status, site_layout, E, W, opers), {"panels": panels}
        dev = ws.device
        groups = _groups(opers, isite, 1)
        nops = len(opers)
        self.E, self.W = E, W
        self.ep = None
        if panels is None:
            panels = torch.device(dev).type == "cuda"
        if panels:
            try:
                self._setup_panels(groups, site_layout, E, W)
                return
            except NoPanelForm:
                pass
        if status == "L":
            ax = (([0], [1]), ([0, 2], [2, 0]), ([1, 3], [1, 0]))
        else:
            ax = (([2], [1]), ([1, 2], [2, 1]), ([1, 3], [1, 2]))
        bases = [numpy.zeros(nops, dtype=numpy.int64) for _ in range(3)]
        tot = [0, 0, 0]
        wbase = numpy.zeros(nops, dtype=numpy.int64)
        wtot = 0
        plans = {}
        out_layouts = [None] * nops
        for key, ops in sorted(groups.items()):
            i0 = ops[0]
            El = E.layouts[i0]
            Wl = W.layouts[i0] if status == "L" else flip_horizontal(W.layouts[i0])
            for i in ops:
                if E.layouts[i] is not El or W.layouts[i] is not W.layouts[i0]:
                    raise ValueError("operators of one symmetry class must share their block structure")
            c1 = Contraction(site_layout, El, ax[0])
            t1 = c1.triples
            c2 = Contraction(Wl, c1.out, ax[1])
            t2 = prune(c2.triples, live2=live_blocks(c1.out, t1))
            c3 = Contraction(c2.out, site_layout, ax[2])
            t3 = prune(c3.triples, live1=live_blocks(c2.out, t2))
            plans[key] = (ops, (c1, t1), (c2, t2), (c3, t3))
            for s, c in enumerate((c1, c2, c3)):
                for i in ops:
                    bases[s][i] = tot[s]
                    tot[s] += c.out.size
                    if s == 2:
                        out_layouts[i] = c.out
        self.out_layouts = out_layouts
        self.out_offsets = bases[2].copy()
        self.tot = tot
        order = numpy.concatenate([numpy.array(plans[k][0]) for k in sorted(plans)])
        tabs = [op_table(0, E.offsets[order], bases[0][order], 1.0),
                op_table(W.offsets[order], bases[0][order], bases[1][order], 1.0),
                op_table(bases[1][order], 0, bases[2][order], 1.0)]
        st = [{}, {}, {}]
        pos = 0
        for key, (ops, *cs) in sorted(plans.items()):
            rng = (pos, pos + len(ops))
            pos += len(ops)
            for si, (c, t) in enumerate(cs):
                add_parts(st[si], compile_classes(c, t, ax[si]), op_range=rng)
        self.stages = [Stage(st[si], dev, "renorm%d" % (si + 1), tabs[si]) for si in range(3)]
        self.flops = sum(s.flops for s in self.stages)

    def _setup_panels(self, groups, site, E, W):
        """The panel form; raises NoPanelForm where the blocks do not allow it."""
        left = self.status == "L"
        old, new = (0, 2) if left else (2, 0)
        if list(site.status) != ([False, False, True] if left else [True, False, False]):
            raise NoPanelForm
        ep = EnvPanels(self.ws, "renorm", groups, site, old, E, W, left, site.qsyms[old], site.qsyms[new])
        dx, dz = ep.dx, ep.dz
        i64 = numpy.int64
        # bra panel of new sector z: [D_z x Kp], K index (x, n') block by block
        o = numpy.lexsort((ep.kn, ep.ky, ep.kz))
        bx, bn, bz = ep.ky[o], ep.kn[o], ep.kz[o]
        cnt = numpy.bincount(bz, minlength=len(dz)).astype(i64)
        first = numpy.cumsum(cnt) - cnt
        Kz = numpy.bincount(bz, weights=dx[bx], minlength=len(dz)).astype(i64)
        ck = numpy.cumsum(dx[bx]) - dx[bx]
        koff = ck - ck[first[bz]]
        Kp = (Kz + 3) // 4 * 4
        boff = numpy.cumsum(dz * Kp) - dz * Kp
        bra = ep._copy_descs(ep.ksrc[o], dx[bx], dz[bz], ep.ket_size + boff[bz] + koff, Kp[bz], old)
        # the new environments' blocks (b, z, z'); T2 panel of each: rows (x, n') of z, columns (b, z')
        wax, sign = (1, 1.0) if left else (0, -1.0)
        lays = [Layout([True, False, True], [sign * wl.qsyms[wax], site.qsyms[new], site.qsyms[new]],
                       [wl.ndims[wax], site.ndims[new], site.ndims[new]]) for wl in ep.Wl]
        sec = [l.block_sectors(l.idx_allowed) for l in lays]
        ok = numpy.repeat(numpy.arange(len(lays)), [len(l.idx_allowed) for l in lays])
        ob, oz, oz2 = (numpy.concatenate([s_[k] for s_ in sec]).astype(i64) for k in range(3))
        ooff = numpy.concatenate([l.ioff[l.idx_allowed] for l in lays])
        ncol = ep.db[ok, ob] * dz[oz2]
        ld = (ncol + 3) // 4 * 4
        size = Kz[oz] * ld
        cs = numpy.cumsum(size) - size
        cls0 = numpy.searchsorted(ok, numpy.arange(len(lays)))
        pan = cs - cs[numpy.minimum(cls0[ok], max(len(cs) - 1, 0))] if len(cs) else cs
        own, loc = _ranges(cnt[oz])
        k = first[oz[own]] + loc                                # bra block of every T2 block
        o2 = pan[own] + koff[k] * ld[own]
        if len(own) and not numpy.array_equal(ep.b[ok[own], bx[k], oz2[own], bn[k]], ob[own]):
            raise NoPanelForm
        ep.finish((ok[own], bx[k], oz2[own], 4 * bn[k], ob[own], o2, ld[own], o2 + dx[bx[k]] * ld[own]),
                  numpy.bincount(ok, weights=size, minlength=len(lays)).astype(i64), bra, int((dz * Kp).sum()))
        base, self._nout = ep.slices([l.size for l in lays], 1)
        u, uj = dpanel_units(ncol, dz[oz], Kz[oz], ld, Kp[oz], pan, boff[oz], ooff, "blk", (dz[oz2], dz[oz]), owner=True)
        nop = numpy.array([len(x) for x in ep.ops])
        fl = 2.0 * float((ncol * dz[oz] * Kz[oz] * nop[ok]).sum())
        self.d3 = DPanelStage("renorm3", ep.by_class(u, ok[uj]), op_table(ep.base_2, 0, base, 1.0), self.ws.device, fl)
        self.out_layouts = [None] * ep.nops
        for l, x in zip(lays, ep.ops):
            for i in x:
                self.out_layouts[i] = l
        self.out_offsets = numpy.empty(ep.nops, dtype=i64)
        self.out_offsets[ep.order] = base
        self.ep = ep
        self.flops = fl + ep.flops1 + (ep.wx.flops if ep.wx is not None else 0.0)

    def __call__(self, site_values):
        """site_values: packed site tensor (float64, device) -> new TensorSet."""
        ws = self.ws
        if self.ep is not None and not self.ep.current():
            self.__init__(*self._args[0], **self._args[1])
        if self.ep is not None:
            out = torch.empty(max(self._nout, 1), dtype=torch.float64, device=ws.device)
            T2, S = self.ep.run(site_values)
            self.d3.run(T2, S[self.ep.ket_size:], out)
            return TensorSet(self.out_layouts, out, self.out_offsets)
        T1 = ws.get("r1", self.tot[0], torch.float64)
        T2 = ws.get("r2", self.tot[1], torch.float64)
        out = torch.zeros(max(self.tot[2], 1), dtype=torch.float64, device=ws.device)
        s = self.stages
        s[0].run(site_values, self.E.values, T1, "f64")
        s[1].run(self.W.values, T1, T2, "f64")
        s[2].run(T2, site_values, out, "f64")
        return TensorSet(self.out_layouts, out, self.out_offsets)


class NoiseRDM(object):
    """Noise term of the decimation's density matrix (pRDMQt with noise > 0).

    status 'L' (source/mpo_dmrg_kernelQt.py:488-531): with psi as [l, n1, X]
    (X = (n2, r) merged), T2_p[l, X, b, n1'] = sum W_p[a, b, n1', n1] L_p[a, l, l'] psi[l', n1, X]
    and rho[l n1', l' n1''] = sum_p sum_{X, b} T2_p T2_p.
    status 'R' (:568-611): with psi as [Y, n2, r] (Y = (l, n1) merged) and R_p flipped,
    T2_p[a, n2', Y, r'] and rho[n2' r', n2'' r''] = sum_p sum_{a, Y} T2_p T2_p.
    Three grouped-GEMM launches over all operators (per-operator Gram blocks), one
    fixed-order sum over operators, and a scatter into the dense matrix the
    decimation uses.  ``psi_layout`` is the rank-3 wavefunction layout (N-reduced
    with spin projection, with qkey[:1] then).
    """

    def __init__(self, ws, isite, status, psi_layout, E, W, opers, qkey, dense_idl, panels=None):
        """panels: the panel form (None: on a GPU, where the blocks allow it): T2 of the module
        envpanels with the rows (l, n1') of one merged class in one panel, whose Gram matrix
        is one panel GEMM of the panel with itself."""
        self.ws, self.status = ws, status
        self._args = (ws, isite, status, psi_layout, E, W, opers, qkey, dense_idl), {"panels": panels}
        dev = ws.device
        groups = _groups(opers, isite, 1)
        nops = len(opers)
        self.E, self.W = E, W
        self.ep = None
        if panels is None:
            panels = torch.device(dev).type == "cuda"
        if panels:
            try:
                self._setup_panels(groups, psi_layout, E, W, qkey, dense_idl)
                return
            except NoPanelForm:
                pass
        if status == "L":
            ax = (([2], [0]), ([0, 2], [0, 3]), ([1, 2], [1, 2]))
        else:
            ax = (([2], [2]), ([1, 3], [2, 1]), ([0, 2], [0, 2]))
        bases = [numpy.zeros(nops, dtype=numpy.int64) for _ in range(2)]
        tot = [0, 0]
        plans = {}
        out = None
        for key, ops in sorted(groups.items()):
            i0 = ops[0]
            El, Wl = E.layouts[i0], W.layouts[i0]
            for i in ops:
                if E.layouts[i] is not El or W.layouts[i] is not Wl:
                    raise ValueError("operators of one symmetry class must share their block structure")
            if status == "L":
                c1 = Contraction(El, psi_layout, ax[0])
                t1 = c1.triples
                c2 = Contraction(c1.out, Wl, ax[1])
                t2 = prune(c2.triples, live1=live_blocks(c1.out, t1))
            else:
                Rl = _flip_right_ket(El, qkey)
                c1 = Contraction(psi_layout, Rl, ax[0])
                t1 = c1.triples
                c2 = Contraction(Wl, c1.out, ax[1])
                t2 = prune(c2.triples, live2=live_blocks(c1.out, t1))
            c3 = Contraction(c2.out, c2.out, ax[2])
            live2 = live_blocks(c2.out, t2)
            t3 = prune(c3.triples, live1=live2, live2=live2)
            if out is None:
                out = c3.out
            elif c3.out is not out:
                raise ValueError("noise RDM blocks differ between operator classes")
            plans[key] = (ops, (c1, t1), (c2, t2), (c3, t3))
            for s, c in enumerate((c1, c2)):
                for i in ops:
                    bases[s][i] = tot[s]
                    tot[s] += c.out.size
        self.out_layout = out
        self.tot = tot
        self.nops = nops
        self.size = out.size if out is not None else 0
        order = numpy.concatenate([numpy.array(plans[k][0]) for k in sorted(plans)])
        slot = numpy.arange(nops, dtype=numpy.int64) * self.size
        if status == "L":
            t0 = op_table(E.offsets[order], 0, bases[0][order], 1.0)
            t1_ = op_table(bases[0][order], W.offsets[order], bases[1][order], 1.0)
        else:
            t0 = op_table(0, E.offsets[order], bases[0][order], 1.0)
            t1_ = op_table(W.offsets[order], bases[0][order], bases[1][order], 1.0)
        tabs = [t0, t1_, op_table(bases[1][order], bases[1][order], slot, 1.0)]
        st = [{}, {}, {}]
        pos = 0
        for key, (ops, *cs) in sorted(plans.items()):
            rng = (pos, pos + len(ops))
            pos += len(ops)
            for si, (c, t) in enumerate(cs):
                add_parts(st[si], compile_classes(c, t, ax[si]), op_range=rng)
        self.stages = [Stage(st[si], dev, "prdm%d" % (si + 1), tabs[si]) for si in range(3)]
        self.flops = sum(s.flops for s in self.stages)
        n = int(numpy.prod(out.shape)) if out is not None else 0
        self.dense_shape = tuple(int(x) for x in out.shape) if out is not None else (0,)
        self.prj = torch.from_numpy(out.prjmap(dense_idl)).to(dev) if out is not None else None
        self.ndense = n

    def _setup_panels(self, groups, psi, E, W, qkey, dense_idl):
        left = self.status == "L"
        if list(psi.status) != [False, False, True]:
            raise NoPanelForm
        i64 = numpy.int64
        qkey = numpy.asarray(qkey, dtype=numpy.float64)
        if left:
            old, qx, qz = 0, psi.qsyms[0], psi.qsyms[2]
        else:           # the right bond's states carry qkey - q(r) in psi, q(r) in the environment
            old, qx, qz = 2, qkey - psi.qsyms[2], qkey - psi.qsyms[0]
        ep = EnvPanels(self.ws, "prdm", groups, psi, old, E, W, left, qx, qz)
        dx, dz = ep.dx, ep.dz
        ncls, nx, nz = len(ep.ops), len(dx), len(dz)
        # merged classes of the rows (x, n'): equal quantum number q(x) + q(n')
        qm = ep.qx[:, None, :] + numpy.rint(2 * psi.qsyms[1]).astype(i64)[None, :, :]
        _, mc = numpy.unique(qm.reshape(nx * 4, -1), axis=0, return_inverse=True)
        mc = mc.ravel()
        nm = int(mc.max()) + 1
        o = numpy.argsort(mc, kind="stable")                    # row blocks (x, n') class by class
        rx, rn, rm = o // 4, o % 4, mc[o]
        K = numpy.bincount(rm, weights=dx[rx], minlength=nm).astype(i64)
        cr = numpy.cumsum(dx[rx]) - dx[rx]
        roff = cr - cr[numpy.searchsorted(rm, rm)]
        # panel of (operator class, merged class): columns (b, z) sector z by sector z
        lead = o[numpy.searchsorted(rm, numpy.arange(nm))]      # any row block of the merged class
        b = ep.b[:, lead // 4, :, lead % 4].transpose(1, 0, 2)  # [class, merged class, z]
        w = numpy.where(b >= 0, ep.db[numpy.arange(ncls)[:, None, None], numpy.maximum(b, 0)] * dz[None, None, :], 0)
        coff = numpy.cumsum(w, axis=2) - w
        wide = w.sum(axis=2)
        ld = (wide + 3) // 4 * 4
        sz = ld * K[None, :]
        pan = numpy.cumsum(sz, axis=1) - sz
        kk, rr, zz = (v.ravel() for v in numpy.nonzero(b[:, rm, :] >= 0))
        m = rm[rr]
        o2 = pan[kk, m] + roff[rr] * ld[kk, m] + coff[kk, m, zz]
        if len(kk) and not numpy.array_equal(ep.b[kk, rx[rr], zz, rn[rr]], b[kk, m, zz]):
            raise NoPanelForm
        ep.finish((kk, rx[rr], zz, 4 * rn[rr], b[kk, m, zz], o2, ld[kk, m], o2 + dx[rx[rr]] * ld[kk, m]),
                  sz.sum(axis=1), numpy.zeros(0, BPERM_DT), 0)
        # Gram matrices: K_m x K_m per merged class, one partial result per operator
        gbase = numpy.cumsum(K * K) - K * K
        self.size = int((K * K).sum())
        self.nops = ep.nops
        rowm, rowi = _ranges(K)
        crow = gbase[rowm] + rowi * K[rowm]
        ck, cm = (v.ravel() for v in numpy.nonzero(numpy.ones((ncls, nm), dtype=bool)))
        r0 = numpy.cumsum(K) - K
        u, uj = dpanel_units(K[cm], K[cm], wide[ck, cm], ld[ck, cm], ld[ck, cm], pan[ck, cm], pan[ck, cm], r0[cm], "row",
                             owner=True)
        fl = 2.0 * float((K[cm] ** 2 * wide[ck, cm] * numpy.array([len(x) for x in ep.ops])[ck]).sum())
        self.d3 = DPanelStage("prdm3", ep.by_class(u, ck[uj]), op_table(ep.base_2, ep.base_2,
                                                                        numpy.arange(ep.nops) * self.size, 1.0),
                              self.ws.device, fl, crow=crow, longest_first=True)
        # dense position of every row: (l, n1) -> 4 l + n1, (n2, r) -> n2 rdim + r
        ix = [numpy.asarray(v, dtype=i64) for v in (dense_idl[0] if left else dense_idl[1])]
        jn = numpy.array([int(v[0]) for v in (dense_idl[1] if left else dense_idl[0])], dtype=i64)
        nxs = int(dx.sum())
        pos = numpy.concatenate([ix[x] * 4 + jn[n] if left else jn[n] * nxs + ix[x] for x, n in zip(rx, rn)])
        d = 4 * nxs
        own, loc = _ranges(K[rowm])
        self.prj = torch.from_numpy(pos[own] * d + pos[r0[rowm[own]] + loc]).to(self.ws.device)
        self.dense_shape = (nxs, 4, nxs, 4) if left else (4, nxs, 4, nxs)
        self.ndense = d * d
        self.ep = ep
        self.flops = fl + ep.flops1 + (ep.wx.flops if ep.wx is not None else 0.0)

    def __call__(self, psi_values):
        """psi_values: packed rank-3 wavefunction (device FP64) -> dense noise RDM (d x d)."""
        ws = self.ws
        if self.ep is not None and not self.ep.current():
            self.__init__(*self._args[0], **self._args[1])
        if self.ep is not None:
            P = ws.get("npart", self.nops * self.size, torch.float64)
            T2, _ = self.ep.run(psi_values)
            self.d3.run(T2, T2, P)
            return self._dense(P)
        T1 = ws.get("n1", self.tot[0], torch.float64)
        T2 = ws.get("n2", self.tot[1], torch.float64)
        P = ws.get("npart", self.nops * self.size, torch.float64)
        s = self.stages
        if self.status == "L":
            s[0].run(self.E.values, psi_values, T1, "f64")
            s[1].run(T1, self.W.values, T2, "f64")
        else:
            s[0].run(psi_values, self.E.values, T1, "f64")
            s[1].run(self.W.values, T1, T2, "f64")
        P[:self.nops * self.size].zero_()
        s[2].run(T2, T2, P, "f64")
        return self._dense(P)

    def _dense(self, P):
        """The sum over operators as the dense matrix the decimation uses."""
        ws = self.ws
        vals = torch.empty(max(self.size, 1), dtype=torch.float64, device=ws.device)[:self.size]
        reduce_ops(P, self.nops, self.size, vals)
        dense = torch.empty(self.ndense, dtype=torch.float64, device=ws.device)
        scatter(vals, self.prj, dense)
        d = self.dense_shape
        return dense.reshape(d[0] * d[1], d[2] * d[3])


def _flip_right_ket(lay, qkey):
    """R environment as pRDMQt 'R' contracts it with the wavefunction's right index
    (kernelQt.py:592-598): qsyms [-q0, -(qkey - q1), qkey - q2], index 1 flipped in/out."""
    st = lay.status.copy()
    st[1] = not st[1]
    qkey = numpy.asarray(qkey, dtype=numpy.float64)
    return Layout(st, [-lay.qsyms[0], -(qkey - lay.qsyms[1]), qkey - lay.qsyms[2]], lay.ndims)
