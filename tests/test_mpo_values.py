"""MPO values as the sparse stages' host builder sees them: what the device holds when the plan is made."""
import numpy
import pytest
import torch

from helpers import load, record_operators, tensorset
from test_sparse_w import _dot, patch


def test_plans_under_inference_mode(monkeypatch):
    """Inference tensors have no version counter; operators are made and run on them as on others."""
    patch(monkeypatch)
    r = load("kernels_K5.npz")["records"][1]
    x = torch.from_numpy(numpy.asarray(r["hvec_x"], dtype=numpy.float64))
    ref = record_operators(r, "cpu", use_fiber=True, fuse_w=False)[0](x)
    with torch.inference_mode():
        y = record_operators(r, "cpu", use_fiber=True, fuse_w=False)[0](x)
        w = tensorset(r["mpo_i"], "cpu")
        w.values[0] += 1.0
        assert w.host()[0] == float(w.values[0])
    assert torch.equal(y, ref)


@pytest.mark.parametrize("what", ["renorm", "noise"])
def test_values_changed_between_plan_and_call(what, monkeypatch):
    """A renormalisation (noise term) made before the MPO was doubled in place, called after it:
    twice (four times) the first result, bit for bit."""
    from helpers import record_noise, record_renormalizer
    from qcmpodmrg_b200 import kernels
    patch(monkeypatch)
    cls = kernels.Renormalizer if what == "renorm" else kernels.NoiseRDM
    make = cls.__init__
    r = next(r for r in load("kernels_%s.npz" % ("K5" if what == "renorm" else "NZ_K5"))["records"]
             if ("renorm_site" if what == "renorm" else "prdm_cimat") in r and numpy.ravel(r["key"])[2] > 0)
    with monkeypatch.context() as m:
        m.setattr(cls, "__init__", lambda self, *a: make(self, *a, panels=True))
        op, vals = (record_renormalizer if what == "renorm" else record_noise)(r, "cpu")[:2]
    vals = torch.as_tensor(vals)
    assert op.ep is not None
    get = (lambda: op(vals).values.clone()) if what == "renorm" else (lambda: op(vals).clone())
    y = get()
    op.W.values.data.mul_(2.0)
    assert torch.equal(get(), (2.0 if what == "renorm" else 4.0) * y) and op.ep is not None


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32", "tf32x3"])
def test_a_write_without_a_trace_is_seen_by_the_next_plan(precision, cuda):
    """The site's MPO doubled through ``.data``: the next plan's product is twice the first one's,
    bit for bit (a power of two)."""
    mk, x = _dot(8, 3, [(4, 0, 8), (3, -1, 3), (5, 1, 2)], [(4, 0, 4), (3, 1, 11), (2, 0, 3)], cuda, precision)
    sig = mk(use_fiber=True, fuse_w=False)
    assert sig.wx is not None
    y = sig(x)
    sig.Wi.values.data.mul_(2.0)
    assert torch.equal(mk(use_fiber=True, fuse_w=False)(x), 2.0 * y)
