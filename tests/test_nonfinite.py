"""An Inf or NaN gets no further through the sparse MPO stage than through the two block contractions."""
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
