"""Tiles of the sparse MPO stage that hold more sector pairs than a tile's tables are cut."""
import numpy
import pytest
import torch

from helpers import load
from test_sparse_w import SECTORS, _dot, patch, sparse_sigma
from qcmpodmrg_b200 import engine


@pytest.mark.parametrize("pairs", [1, 2])
@pytest.mark.parametrize("tag", ["K5", "K6"])
def test_cut_tiles(tag, pairs, monkeypatch):
    """The reference's products with tiles of at most ``pairs`` sector pairs (the interpreter checks
    the limit and that every element is written once)."""
    patch(monkeypatch)
    cut = 0
    for r in load("kernels_%s.npz" % tag)["records"]:
        whole = sparse_sigma(r, "cpu")
        with monkeypatch.context() as m:
            m.setattr(engine, "WX_GRPS", pairs)
            sig = sparse_sigma(r, "cpu")
            if sig.wx is None:
                continue
            cut += len(sig.wx.items("f64")[0][1]) > len(whole.wx.items("f64")[0][1])
            y = sig(torch.from_numpy(numpy.asarray(r["hvec_x"], dtype=numpy.float64))).numpy()
        ref = numpy.asarray(r["hvec_y"])
        assert numpy.abs(y - ref).max() <= 1e-12 * max(1.0, numpy.abs(ref).max())
    assert cut


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_cut_tiles_on_the_device(precision, cuda, monkeypatch):
    """Bit for bit the products of whole tiles: a cut changes no sum."""
    nl, nr = SECTORS[3]
    mk, x = _dot(8, 3, nl, nr, cuda, precision)
    ref = mk(use_fiber=True, fuse_w=False)(x)
    for pairs in (1, 2):
        monkeypatch.setattr(engine, "WX_GRPS", pairs)
        assert torch.equal(mk(use_fiber=True, fuse_w=False)(x), ref)
