"""The diagonal's panel tasks cut their operators to the extent of a launch's grid."""
import numpy
import pytest
import torch

from helpers import load, record_operators
from test_sparse_w import patch
from qcmpodmrg_b200 import kernels


def test_ranges_fit_the_grid():
    """5000 operators (spin projection: spin orbitals times quadrature points), 16 tasks each."""
    stages = kernels._diag_stages(torch.device("cpu"), 5000, 1, 1, 1, 2, 2, numpy.ones(5000))
    for st, count in zip(stages, (80000, 80000, 16)):
        seen = []
        for _, tk, _, span in st.groups:
            assert span <= 65535 and int((tk["op_e"] - tk["op_b"]).max()) <= 65535
            seen += [i for t in tk for i in range(t["op_b"], t["op_e"])]
        assert sorted(seen) == list(range(count))


@pytest.mark.parametrize("tag", ["K4", "K5"])
def test_cut_ranges_give_the_same_diagonal(tag, monkeypatch):
    """Bit for bit: every product is one task's, in the same order."""
    patch(monkeypatch)
    for r in load("kernels_%s.npz" % tag)["records"][:3]:
        ref = record_operators(r, "cpu")[1]().clone()
        with monkeypatch.context() as m:
            m.setattr(kernels, "PANEL_OPS", 7)
            m.setattr(kernels, "_DENSE_STAGES", {})
            assert torch.equal(record_operators(r, "cpu")[1](), ref)
