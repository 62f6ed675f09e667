"""Renormalisation and noise term in panel form: tensors whose contracted indices do not match are
refused, as by the block contractions, and MPO bonds with a repeated quantum number keep those."""
import numpy
import pytest
import torch

from helpers import load, record_noise, record_renormalizer
from test_sparse_w import patch
from qcmpodmrg_b200 import kernels
from qcmpodmrg_b200.kernels import TensorSet
from qcmpodmrg_b200.qtensor import Layout


def _swapped(lay, axis):
    """The layout with two equally large sectors of one index exchanged (None: it has none)."""
    n = lay.ndims[axis]
    for i in range(len(n)):
        for j in range(i):
            if n[i] == n[j]:
                q = [numpy.array(v) for v in lay.qsyms]
                q[axis][[i, j]] = q[axis][[j, i]]
                return Layout(lay.status, q, lay.ndims)
    return None


def _args(what, status, monkeypatch):
    """Constructor arguments of a recorded renormalisation or noise term."""
    cls, rec, tag = {"renorm": (kernels.Renormalizer, record_renormalizer, "K6"),
                     "noise": (kernels.NoiseRDM, record_noise, "NZ_K6")}[what]
    key = "renorm_site" if what == "renorm" else "prdm_cimat"
    got = []
    with monkeypatch.context() as m:
        m.setattr(cls, "__init__", lambda self, *a, **k: got.append(a))
        for r in load("kernels_%s.npz" % tag)["records"]:
            if key in r and numpy.ravel(r["key"])[1] == (status == "R"):
                rec(r, "cpu")
    return cls, list(got[0])


@pytest.mark.parametrize("status", ["L", "R"])
@pytest.mark.parametrize("what", ["renorm", "noise"])
@pytest.mark.parametrize("where", ["site", "E0", "E2", "W"])
def test_exchanged_sectors_are_refused(what, status, where, monkeypatch):
    patch(monkeypatch)
    cls, a = _args(what, status, monkeypatch)
    ws, isite, st, site, E, W = a[:6]
    cls(*a, panels=True)
    left = status == "L"
    if where == "site":
        a[3] = _swapped(site, 0 if left else 2)
        if a[3] is None:
            pytest.skip("no two sectors of one size")
    else:
        t, axis = (W, 0 if left else 1) if where == "W" else (E, int(where[1]))
        lays = {id(l): _swapped(l, axis) for l in t.layouts}
        if any(v is None for v in lays.values()):
            pytest.skip("no two sectors of one size")
        a[5 if where == "W" else 4] = TensorSet([lays[id(l)] for l in t.layouts],
                                                torch.zeros(sum(v.size for v in t.layouts) * 2, dtype=torch.float64))
    for panels in (True, False):
        with pytest.raises(ValueError):
            cls(*a, panels=panels)


@pytest.mark.parametrize("status", ["L", "R"])
@pytest.mark.parametrize("what", ["renorm", "noise"])
def test_a_repeated_sector_keeps_the_block_contractions(what, status, monkeypatch):
    """The open MPO bond's largest sector given as two of the same quantum number: the values of the
    block contractions."""
    patch(monkeypatch)
    cls, a = _args(what, status, monkeypatch)
    W = a[5]
    axis = 1 if status == "L" else 0
    rng = numpy.random.default_rng(5)
    lays = {}
    for l in W.layouts:
        k = int(numpy.argmax(l.ndims[axis]))
        n, q = list(l.ndims), list(l.qsyms)
        n[axis] = numpy.insert(n[axis], k, 1)
        q[axis] = numpy.insert(q[axis], k, q[axis][k], axis=0)
        lays[id(l)] = Layout(l.status, q, n)
    new = [lays[id(l)] for l in W.layouts]
    a[5] = TensorSet(new, [rng.standard_normal(l.size) for l in new], device="cpu")
    x = torch.from_numpy(rng.standard_normal(a[3].size))
    y, ref = (op(x) if what == "noise" else op(x).values for op in (cls(*a, panels=p) for p in (True, False)))
    assert torch.equal(y, ref)


def test_scratch_is_not_shared(monkeypatch):
    """A renormalisation and a noise term on one workspace use different buffers, as their block
    contractions do, so that one may run beside the other on a stream of its own."""
    patch(monkeypatch)
    names = []
    for what in ("renorm", "noise"):
        cls, a = _args(what, "L", monkeypatch)
        op = cls(*a, panels=True)
        op(torch.zeros(a[3].size, dtype=torch.float64))
        assert op.ep is not None
        names.append(set(a[0].bufs))
    assert names[0] and names[1] and not names[0] & names[1]
