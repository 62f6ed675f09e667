"""One environment contracted with a rank-3 tensor and an MPO site, in panel form.

Renormalisation (renormQt_H00, source/mpo_dmrg_kernelQt.py:633-767) and the noise term of
the density matrix (pRDMQt, :453-626) share their first two contractions:

  T1[a, x, n, z] = sum_y E[a, x, y] S[y, n, z]                 (panel GEMM, k_dpanel)
  T2[b, n', (x, z)] = sum_{a, n} W[a, b, n', n] T1[a, x, n, z]  (sparse product, k_wsparse)

with E the environment (MPO bond a, bra and ket states x, y of the old bond), S the site
tensor or the wavefunction with one physical and one new index, and W the site's MPO (from
the right, with its bonds exchanged).  E and S become K-major panels per sector y by block
copies; the blocks of T2 go where the caller's last contraction wants them.  The plan is
built for all operator classes in one pass of array operations.
"""
import numpy
import torch

from .engine import (BPERM_DT, DCOL_DT, DPanelStage, SparseWStage, WSource, dpanel_units, op_table, sparse_groups,
                     upload, _ranges)

i64 = numpy.int64


def _pad(n, q):
    return (n + q - 1) // q * q


def _q2(q):
    return numpy.rint(2 * numpy.asarray(q, dtype=numpy.float64)).astype(i64)


class NoPanelForm(Exception):
    """The blocks of these tensors have no panel form (the grouped block GEMM takes them)."""


class EnvPanels(object):
    """Stages 1 and 2 for every operator; see the module's docstring.

    groups: {class: operators}; site: layout of S as its packed values are stored; old: its
    contracted axis (0 or 2); left: W's input bond is its left one; qx, qz: quantum numbers
    of the old and new bond's sectors with q(a) = q(x) - q(y), q(z) = q(y) + q(n)."""

    def __init__(self, ws, name, groups, site, old, E, W, left, qx, qz):
        self.ws, self.name, self.E = ws, name, E
        self.keys = sorted(groups)
        self.ops = [groups[k] for k in self.keys]
        self.order = numpy.concatenate([numpy.asarray(o) for o in self.ops])
        ends = numpy.cumsum([len(o) for o in self.ops])
        self.ranges = [(int(e) - len(o), int(e)) for o, e in zip(self.ops, ends)]
        self.nops = int(ends[-1])
        self.El = [E.layouts[o[0]] for o in self.ops]
        self.Wl = [W.layouts[o[0]] for o in self.ops]
        for o, el, wl in zip(self.ops, self.El, self.Wl):
            if any(E.layouts[i] is not el or W.layouts[i] is not wl for i in o):
                raise ValueError("operators of one symmetry class must share their block structure")
        new = 2 - old
        if site.rank != 3 or len(site.ndims[1]) != 4 or (site.ndims[1] != 1).any() or not len(site.idx_allowed):
            raise NoPanelForm
        qn = _q2(site.qsyms[1])
        for el, wl in zip(self.El, self.Wl):
            if list(el.status) != [True, False, True] or list(wl.status) != [False, True, False, True]:
                raise NoPanelForm
            for k in (2, 3):
                if len(wl.ndims[k]) != 4 or (wl.ndims[k] != 1).any() or not numpy.array_equal(_q2(wl.qsyms[k]), qn):
                    raise NoPanelForm
        dx, dz = (numpy.asarray(site.ndims[k], dtype=i64) for k in (old, new))
        self.dx, self.dz = dx, dz
        # contracted indices have the same sectors in the same order (the block contractions, which take
        # what does not, refuse other ones): E's bond states those of S, its MPO bond W's
        wk, sign = (0, 1) if left else (1, -1)

        def same(mine, theirs, number=numpy.asarray):
            return [len(v) for v in mine] == [len(v) for v in theirs] and \
                numpy.array_equal(number(numpy.concatenate(mine)), number(numpy.concatenate(theirs)))

        bonds = [(el, k) for el in self.El for k in (1, 2)]
        if not (same([el.ndims[k] for el, k in bonds], [dx] * len(bonds))
                and same([el.qsyms[k] for el, k in bonds], [qx] * len(bonds), _q2)
                and same([el.ndims[0] for el in self.El], [wl.ndims[wk] for wl in self.Wl])
                and same([sign * el.qsyms[0] for el in self.El], [wl.qsyms[wk] for wl in self.Wl], _q2)):
            raise NoPanelForm
        ncls, nx, nz = len(self.ops), len(dx), len(dz)
        # ---- S: blocks sorted by contracted sector, side by side as the columns of its panel
        sec = site.block_sectors(site.idx_allowed)
        y, n, z = (numpy.asarray(sec[k], dtype=i64) for k in (old, 1, new))
        o = numpy.argsort(y, kind="stable")
        y, n, z, src = y[o], n[o], z[o], site.ioff[site.idx_allowed][o]
        self.ky, self.kn, self.kz, self.ksrc = y, n, z, src
        N = dz[z]
        cnt = numpy.bincount(y, minlength=nx).astype(i64)
        kfirst = numpy.cumsum(cnt) - cnt
        ntot = numpy.bincount(y, weights=N, minlength=nx).astype(i64)
        cn = numpy.cumsum(N) - N
        col = cn - cn[kfirst[y]]
        col0 = numpy.cumsum(ntot) - ntot
        ncol = int(ntot.sum())
        kp = _pad(dx, 4)
        soff = numpy.cumsum(ntot * kp) - ntot * kp
        self.ket_size = int((ntot * kp).sum())
        self.ket_descs = self._copy_descs(src, dx[y], N, soff[y] + col * kp[y], kp[y], old)
        # ---- E: rows (a, x) of every contracted sector y, stacked per class
        ek, ea, ex, ey, eoff = [], [], [], [], []
        for k, el in enumerate(self.El):
            a, x, yy = el.block_sectors(el.idx_allowed)
            ek.append(numpy.full(len(a), k, dtype=i64))
            ea.append(a)
            ex.append(x)
            ey.append(yy)
            eoff.append(el.ioff[el.idx_allowed])
        ek, ea, ex, ey, eoff = (numpy.concatenate(v).astype(i64) for v in (ek, ea, ex, ey, eoff))
        keep = cnt[ey] > 0
        ek, ea, ex, ey, eoff = (v[keep] for v in (ek, ea, ex, ey, eoff))
        o = numpy.argsort(ek * nx + ey, kind="stable")
        ek, ea, ex, ey, eoff = (v[o] for v in (ek, ea, ex, ey, eoff))
        na = max(max(len(el.ndims[0]) for el in self.El), 1)
        da = numpy.zeros((ncls, na), dtype=i64)
        for k, el in enumerate(self.El):
            da[k, :len(el.ndims[0])] = el.ndims[0]
        rows = da[ek, ea] * dx[ex]
        ky = ek * nx + ey
        M = numpy.bincount(ky, weights=rows, minlength=ncls * nx).astype(i64)
        cr = numpy.cumsum(rows) - rows
        rowoff = cr - cr[numpy.searchsorted(ky, ky)] if len(ky) else cr
        lsz = (M.reshape(ncls, nx) * kp[None, :])
        lpoff = (numpy.cumsum(lsz, axis=1) - lsz).ravel()
        d = numpy.zeros(len(ek), BPERM_DT)
        d["src_off"], d["dst_off"] = eoff, lpoff[ky] + rowoff * kp[ey]
        d["d0"], d["d1"], d["d2"] = da[ek, ea], dx[ex], dx[ey]
        d["s0"], d["s1"], d["s2"] = dx[ex] * kp[ey], kp[ey], 1
        rng = numpy.array(self.ranges, dtype=i64).reshape(-1, 2)
        d["op_b"], d["op_e"] = rng[ek, 0], rng[ek, 1]
        self.env_descs = d
        # ---- T1: one panel [M x N_j] per class and block of S
        tsz = M.reshape(ncls, nx)[:, y] * N[None, :]
        t1pan = numpy.cumsum(tsz, axis=1) - tsz
        own, loc = _ranges(cnt[ey])
        j = kfirst[ey[own]] + loc
        o1 = t1pan[ek[own], j] + rowoff[own] * N[j]
        self._ins = (ek[own], ex[own], z[j], 4 * n[j], ea[own], o1, None, o1 + rows[own] * N[j])
        if max(int(tsz.sum(axis=1).max()), int(lsz.sum(axis=1).max())) >= 2 ** 31:
            raise NoPanelForm
        own, loc = _ranges(N)
        tab = numpy.zeros((ncls, max(ncol, 1)), DCOL_DT)
        tab["off"] = t1pan[:, own] + loc[None, :]
        tab["ld"] = N[own][None, :]
        pk, py = (v.ravel() for v in numpy.nonzero((M.reshape(ncls, nx) > 0) & (ntot > 0)[None, :]))
        u, uj = dpanel_units(M[pk * nx + py], ntot[py], dx[py], kp[py], kp[py], lpoff[pk * nx + py], soff[py],
                             pk * max(ncol, 1) + col0[py], "col", owner=True)
        self.parts1 = self.by_class(u, pk[uj])
        self.cols = tab.ravel()
        self.flops1 = 2.0 * float((M[pk * nx + py] * ntot[py] * dx[py] *
                                   numpy.array([len(o) for o in self.ops])[pk]).sum())
        self.base_e, self.tot_e = self.slices(lsz.sum(axis=1))
        self.base_1, self.tot_1 = self.slices(tsz.sum(axis=1))
        # ---- T2: the output sector b of every (class, x, z, n')
        wax = 1 if left else 0
        sign = 1 if left else -1
        nb = max(max(len(wl.ndims[wax]) for wl in self.Wl), 1)
        self.db = numpy.zeros((ncls, nb), dtype=i64)
        self.qx, self.qz = _q2(qx), _q2(qz)
        want = (self.qx[:, None, None, :] - self.qz[None, :, None, :] + qn[None, None, :, :])    # [x, z, n', q]
        self.b = numpy.full((ncls, nx, nz, 4), -1, dtype=i64)
        # quantum numbers as one integer each; the largest absolute value bounds every digit
        qw = [sign * _q2(wl.qsyms[wax]) for wl in self.Wl]
        top = max([int(abs(want).max())] + [int(abs(q).max()) for q in qw if len(q)])
        code = lambda q: (q + top) @ ((2 * top + 1) ** numpy.arange(q.shape[-1], dtype=i64))          # noqa: E731
        cw = code(want)
        for k, (wl, q) in enumerate(zip(self.Wl, qw)):
            if len(q) == 0:
                continue
            self.db[k, :len(q)] = wl.ndims[wax]
            cq = code(q)
            o = numpy.argsort(cq, kind="stable")
            if (numpy.diff(cq[o]) == 0).any():          # two sectors of one quantum number
                raise NoPanelForm
            at = o[numpy.minimum(numpy.searchsorted(cq[o], cw), len(q) - 1)]
            self.b[k] = numpy.where(cq[at] == cw, at, -1)
        self._w = (W, left, wax, qx, qz, da)

    @staticmethod
    def _copy_descs(src, d_old, d_new, dst, stride, old):
        """Copies of packed blocks of S (old and new index in storage order) to K-major rows:
        (old, new) -> dst + old + new * stride."""
        d = numpy.zeros(len(src), BPERM_DT)
        d["src_off"], d["dst_off"] = src, dst
        d["d0"] = 1
        if old == 0:
            d["d1"], d["d2"], d["s1"], d["s2"] = d_old, d_new, 1, stride
        else:
            d["d1"], d["d2"], d["s1"], d["s2"] = d_new, d_old, stride, 1
        d["op_e"] = 1
        return d

    def by_class(self, units, cls):
        """[(units, operator range)] of units sorted by class."""
        cut = numpy.searchsorted(cls, numpy.arange(len(self.ops) + 1))
        return [(units[cut[k]:cut[k + 1]], r) for k, r in enumerate(self.ranges) if cut[k + 1] > cut[k]]

    def slices(self, sizes, align=32):
        """(first element of every operator's slice, total) for per-class slice sizes."""
        sz = numpy.repeat(_pad(numpy.asarray(sizes, dtype=i64), align), [len(o) for o in self.ops])
        return numpy.cumsum(sz) - sz, int(sz.sum())

    def finish(self, outs, sizes, extra_descs, extra_size):
        """The stages, with T2 block (class, x, z, n') -> outs (sparse_groups' form) in slices of
        the given per-class sizes; extra_descs: further copies of S's blocks, behind the ket
        panels (extra_size elements)."""
        dev = self.ws.device
        W, left, wax, qx, qz, da = self._w
        parts = sparse_groups(self._ins, outs, self.dx, self.dz, qx, qz, da, self.db)
        if parts is None or max(int(s) for s in sizes) >= 2 ** 31:
            raise NoPanelForm
        self.base_2, self.tot_2 = self.slices(sizes)
        # compared with the device when the plan runs (current): comparing here would wait for the
        # stream while the rows are still to be made (renormalisations back to back, K=24, D=500:
        # 11.2 instead of 9.0 ms)
        w = W.host(check=False)
        self._mpo = (W, w)
        if not W.finite(w):
            raise NoPanelForm
        source = WSource.of if left else WSource.transposed
        values = w if left else W.transposed(w)
        wp = []
        for k, (g, rng) in enumerate(zip(parts, self.ranges)):
            if g is None:
                continue
            f = source(self.Wl[k], values, W.offsets[self.ops[k]])
            wp.append((g, rng, (f, WSource.identity(self.Wl[k].ndims[wax], rng[1] - rng[0]))))
        z = numpy.zeros(self.nops, dtype=i64)
        self.wx = SparseWStage(wp, dev, self.name + "2", op_table(self.base_1, 0, self.base_2, 1.0)) if wp else None
        self.d1 = DPanelStage(self.name + "1", self.parts1, op_table(self.base_e, z, self.base_1, 1.0), dev, self.flops1,
                              cols=self.cols)
        self.site_descs = numpy.concatenate([self.ket_descs, extra_descs])
        self.site_size = self.ket_size + extra_size
        one = op_table(0, 0, 0, 1.0)
        self._site_d, self._env_d = upload(self.site_descs, dev), upload(self.env_descs, dev)
        self._one = upload(one, dev)
        self._env_ops = upload(op_table(self.E.offsets[self.order], 0, self.base_e, 1.0), dev)
        self._span = max(len(o) for o in self.ops)
        self._ins = self._w = None

    def current(self):
        """Whether the MPO still has the values that the plan was made from (not known, and taken
        as true, while a graph is captured)."""
        W, w = self._mpo
        if W.values.is_cuda and torch.cuda.is_current_stream_capturing():
            return True
        now = W.host()
        return now is w or numpy.array_equal(now, w)

    def run(self, values):
        """T2 and the panels of S for the packed values of S."""
        from . import kernels as K
        # scratch of its own for each kind of contraction: a noise term may run beside a renormalisation
        get = lambda name, n: self.ws.get(self.name + name, n, torch.float64)          # noqa: E731
        S, EP = get("_site", self.site_size), get("_env", self.tot_e)
        T1, T2 = get("_t1", self.tot_1), get("_t2", self.tot_2)
        K.block_permute(self._site_d, len(self.site_descs), 1, self._one, values, S)
        K.block_permute(self._env_d, len(self.env_descs), self._span, self._env_ops, self.E.values, EP)
        self.d1.run(EP, S, T1)
        if self.wx is not None:
            self.wx.run(T1, None, T2, "f64")
        return T2, S
