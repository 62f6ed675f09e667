"""FP32 and split-TF32 products of operators that were made for FP64 (HVec's ``precision`` argument,
lockstep batches of FP64 instances): their sparse stage derives its coefficients from the FP64 ones."""
import numpy
import pytest
import torch

from helpers import load
from test_sparse_w import SECTORS, _dot, patch, sparse_sigma


@pytest.mark.parametrize("tag", ["K4", "K5", "K5N2"])
def test_derived_coefficients_are_the_compiled_ones(tag, monkeypatch):
    """Bit for bit, on the host and on the device; the work items are the FP64 plan's."""
    patch(monkeypatch)
    used = 0
    for r in load("kernels_%s.npz" % tag)["records"]:
        a, b = sparse_sigma(r, "cpu"), sparse_sigma(r, "cpu", precision="f32")
        if a.wx is None:
            continue
        used += 1
        ref = b.wx.h_w["f32"]
        assert numpy.array_equal(a.wx.host_weights("f32"), ref)
        assert numpy.array_equal(a.wx.weights("f32").numpy(), ref)
        assert a.wx.items("f32") is a.wx.items("f64")
    assert used


@pytest.mark.gpu
@pytest.mark.parametrize("case", range(len(SECTORS)))
def test_products(case, cuda):
    """FP32's 2e-5 of the FP64 product, as for operators made for FP32; also in a captured graph."""
    nl, nr = SECTORS[case]
    mk, x = _dot(8, 3, nl, nr, cuda, "f64")
    ref = mk(use_fiber=False, panel1=False)(x)
    tol = 2e-5 * float(torch.linalg.norm(ref))
    for precision in ("f32", "tf32", "tf32x3"):
        sig = mk(use_fiber=True, fuse_w=False)
        assert sig.wx is not None
        for _ in range(2):
            assert float(torch.linalg.norm(sig(x, precision=precision) - ref)) <= tol
    # an operator whose first FP32 product is captured: its panels and coefficients are made by the replay
    sig, y = mk(use_fiber=True, fuse_w=False), torch.empty_like(ref)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sig(x, y, precision="f32")
    g.replay()
    assert float(torch.linalg.norm(y - ref)) <= tol


@pytest.mark.gpu
def test_lockstep_batch(cuda):
    from qcmpodmrg_b200.batched import BatchedSigma
    sigs, xs = zip(*((mk(use_fiber=True, fuse_w=False), x)
                     for mk, x in (_dot(8, 3, nl, nr, cuda, "f64") for nl, nr in SECTORS)))
    for y, s, x in zip(BatchedSigma(list(sigs), cuda, "f32")(list(xs)), sigs, xs):
        ref = s(x)
        assert float(torch.linalg.norm(y - ref)) <= 2e-5 * float(torch.linalg.norm(ref))
