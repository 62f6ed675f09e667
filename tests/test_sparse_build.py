"""The host builder of the sparse MPO stage: exchanged bonds and concurrent builds."""
from concurrent.futures import ThreadPoolExecutor

import numpy
import pytest
import torch

from helpers import load, record_renormalizer, tensorset
from test_sparse_w import patch, sparse_sigma
from qcmpodmrg_b200 import kernels


def test_transposed_values():
    """Every block of every operator, transposed in its place."""
    for r in load("kernels_K5.npz")["records"][:3]:
        w = tensorset(r["mpo_i"], "cpu")
        t = w.transposed(w.host())
        for lay, o in zip(w.layouts, w.offsets):
            for b in lay.idx_allowed:
                d = lay.block_dims(numpy.array([b]))[0]
                s = slice(int(o) + int(lay.ioff[b]), int(o) + int(lay.ioff[b]) + int(numpy.prod(d)))
                assert numpy.array_equal(t[s].reshape(d[1], d[0]), w.host()[s].reshape(d[0], d[1]).T)


def test_bonds_are_exchanged_once(monkeypatch):
    """Renormalisations from the right share one exchanged copy of the site's values, and a changed
    site gets its own."""
    patch(monkeypatch)
    calls, make = [], kernels.transposed_values
    monkeypatch.setattr(kernels, "transposed_values", lambda *a: calls.append(1) or make(*a))
    r = next(r for r in load("kernels_K5.npz")["records"] if "renorm_site" in r and numpy.ravel(r["key"])[1] == 1)
    init = kernels.Renormalizer.__init__
    monkeypatch.setattr(kernels.Renormalizer, "__init__",
                        lambda self, *a, **k: init(self, *a, **dict({"panels": True}, **k)))
    rn, site = record_renormalizer(r, "cpu")
    assert rn.ep is not None
    y = rn(torch.from_numpy(site)).values.clone()
    again = kernels.Renormalizer(*rn._args[0])
    assert torch.equal(again(torch.from_numpy(site)).values, y) and len(calls) == 1
    rn.W.values.mul_(2.0)
    assert torch.equal(again(torch.from_numpy(site)).values, 2.0 * y) and len(calls) == 2


def test_concurrent_builds(monkeypatch):
    """Plans made by eight threads at once are those of one thread, byte for byte."""
    monkeypatch.setattr(kernels, "block_permute", lambda *a: None)
    recs = load("kernels_K6.npz")["records"][:4]
    ref = [_tables(r) for r in recs]
    assert any(ref)
    with ThreadPoolExecutor(8) as pool:
        assert list(pool.map(_tables, recs * 8)) == ref * 8


def _tables(r):
    wx = sparse_sigma(r, "cpu", precision="f32").wx
    if wx is None:
        return []
    return [getattr(wx, n).tobytes() for n in ("h_dops", "h_octs", "h_ent_r", "h_groups", "h_deltas", "h_rows")] + \
        [wx.h_w[k].tobytes() for k in ("f64", "f32")]


def test_sites_of_different_bonds_are_refused():
    """The second site's left bond one state shorter than the first one's right bond."""
    from qcmpodmrg_b200 import engine, native
    ones, four = numpy.ones(1, dtype=numpy.int64), numpy.ones(4, dtype=numpy.int64)

    def source(a, b):
        return engine.WSource(numpy.ones(16 * a * b), [0], [1, 1, 4, 4], numpy.concatenate([a * ones, b * ones, four, four]),
                              numpy.arange(16) * a * b, numpy.ones(16))

    i32 = numpy.int32
    part = {"groups": numpy.zeros(1, engine.WXGRP_DT), "deltas": numpy.zeros(1, engine.WXDELTA_DT),
            "rows": numpy.zeros(2, i32), "fibers": numpy.ones(1, dtype=numpy.int64),
            "iblk": numpy.array([[0] + [-1] * 15], i32), "kblk": numpy.array([[0] + [-1] * 15], i32),
            "row0": numpy.zeros((1, 16), i32), "R": numpy.array([2], i32)}
    part["deltas"]["R"], part["deltas"]["grp_e"] = 2, 1
    make = lambda b: engine.SparseWStage([(part, (0, 1), (source(2, 3), source(b, 2)))], "cpu", "s",            # noqa: E731
                                         engine.op_table(0, 0, 0, 1.0))
    assert len(make(3).h_octs) == 1
    with pytest.raises(native.NativeError):
        make(2)
