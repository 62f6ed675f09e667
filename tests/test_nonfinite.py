"""An Inf or NaN gets no further through the sparse MPO stage than through the block contractions."""
import numpy
import pytest
import torch

from helpers import load
from test_sparse_w import interpret, patch, sparse_sigma


@pytest.mark.parametrize("tag", ["K4", "K6"])
def test_a_bad_element_of_t1(tag, monkeypatch):
    """Every T1 element in turn (a sample of 12): the T3 elements that turn non-finite are among
    those that the separate stages, which multiply by the zeros inside their W panels, give."""
    patch(monkeypatch)
    rng = numpy.random.default_rng(4)
    used = 0
    for r in load("kernels_%s.npz" % tag)["records"]:
        sig = sparse_sigma(r, "cpu")
        if sig.wx is None:
            continue
        used += 1
        n = sig.tot[0] + 64
        clean = torch.from_numpy(rng.standard_normal(n))
        new, old, T2 = (torch.zeros(sig.tot[k] + 64, dtype=torch.float64) for k in (2, 2, 1))
        for at in rng.choice(sig.tot[0], min(12, sig.tot[0]), replace=False):
            T1 = clean.clone()
            T1[at] = float("nan") if at % 2 else float("inf")
            new.zero_(), old.zero_(), T2.zero_()
            with numpy.errstate(invalid="ignore"):
                interpret(sig.wx, T1, new)
                sig.stages[1].run(T1, sig.Wi.values, T2, "f64")
                sig.stages[2].run(T2, sig.Wj.values, old, "f64")
            bad, may = ~torch.isfinite(new), ~torch.isfinite(old)
            assert not bool((bad & ~may).any())
    assert used


@pytest.mark.parametrize("at, bad", [(40, float("nan")), (120, float("inf"))])
def test_a_bad_element_of_the_mpo(at, bad, monkeypatch):
    """Operators of such an MPO keep the block contractions: the same non-finite elements, products,
    environments and noise terms alike."""
    from helpers import record_noise, record_renormalizer, tensorset
    from qcmpodmrg_b200 import kernels
    patch(monkeypatch)

    def spoilt(dicts, device):
        w = tensorset(dicts, device)
        if len(w.layouts[0].nsyms) == 4:
            nz = torch.nonzero(w.values).ravel()
            w.values[nz[at % len(nz)]] = bad
        return w

    monkeypatch.setattr("helpers.tensorset", spoilt)
    monkeypatch.setattr("test_sparse_w.tensorset", spoilt)

    def both(cls, name, run):
        make, out = cls.__init__, []
        for on in (True, False):
            with monkeypatch.context() as m, numpy.errstate(invalid="ignore"):
                m.setattr(cls, "__init__", lambda self, *a, **k: make(self, *a, **dict({name: on}, **k)))
                out.append(run())
        return out

    r = next(r for r in load("kernels_K5.npz")["records"] if numpy.ravel(r["key"])[2] == 1 and "renorm_site" in r)
    x = torch.from_numpy(numpy.asarray(r["hvec_x"], dtype=numpy.float64))
    a, b = (sparse_sigma(r, "cpu", on)(x) for on in (True, False))
    assert not bool(torch.isfinite(b).all()) and torch.equal(torch.isfinite(a), torch.isfinite(b))

    def renorm():
        op, site = record_renormalizer(r, "cpu")
        return op(torch.from_numpy(site)).values

    a, b = both(kernels.Renormalizer, "panels", renorm)
    assert not bool(torch.isfinite(b).all()) and torch.equal(torch.isfinite(a), torch.isfinite(b))
    rn = next(r for r in load("kernels_NZ_K5.npz")["records"] if "prdm_cimat" in r and numpy.ravel(r["key"])[2] == 1)

    def noise():
        op, vals = record_noise(rn, "cpu")[:2]
        return op(torch.as_tensor(vals))

    a, b = both(kernels.NoiseRDM, "panels", noise)
    assert not bool(torch.isfinite(b).all()) and torch.equal(torch.isfinite(a), torch.isfinite(b))
