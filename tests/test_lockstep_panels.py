"""Operators of lockstep batches hold the row-major panels only, until a product runs on its own."""
import numpy
import pytest
import torch

from helpers import load
from test_sparse_w import patch
from qcmpodmrg_b200.dmrg import DMRG
from qcmpodmrg_b200.hamiltonian import make_hamiltonian


def _run(device, precision):
    fx = load("sweep_K6.npz")
    ham = make_hamiltonian(int(fx["K"]), int(fx["N"]), int(fx["seed"]), None if fx["decay"] < 0 else fx["decay"])
    d = DMRG(ham, device=device, precision=precision)
    d.sigma_opts["sparse_w"] = True
    d.load_mps(fx["init_mps"])
    d.sweep("R", int(fx["D"]), 1e-8)
    d.psi0 = None               # (the start vector of the next sweep's first dot, not of the one below)
    return d


def _check(d):
    ctx = d.dot_begin(2, 1e-8)
    sig = ctx["sig"]
    assert sig.wx is not None
    names = ["lpan64", "rpan64", "lpan_f32", "rpan_f32", "lpan_tc", "rpan_tc"]
    assert all(getattr(sig, n) is None for n in names)
    x = torch.from_numpy(numpy.random.default_rng(1).standard_normal(sig.ndim0)).to(d.device)
    y = sig(x).clone()
    assert sig.lpan64 is not None and sig.rpan64 is not None
    d.plan_cache.clear()
    ref = d.dot_operators(2)[2]
    assert ref.lpan64 is not None and torch.equal(ref(x), y)
    # the same plan, reused for the other purpose and back
    assert d.dot_begin(2, 1e-8)["sig"] is ref and all(getattr(ref, n) is None for n in names)
    assert d.dot_operators(2)[2] is ref and ref.lpan64 is not None and torch.equal(ref(x), y)


def test_panels_are_made_by_the_first_product(monkeypatch):
    patch(monkeypatch)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a, **k: None)
    _check(_run("cpu", "f64"))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["f64", "f32", "tf32x3"])
def test_on_the_device(precision, cuda):
    _check(_run(cuda, precision))
