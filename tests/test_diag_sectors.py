"""The diagonal reads every MPO bond sector of quantum number zero."""
import numpy
import pytest
import torch

from helpers import layout_of, load, tensorset
from test_sparse_w import patch
from qcmpodmrg_b200.kernels import DiagOperator, TensorSet, Workspace
from qcmpodmrg_b200.qtensor import Layout


def _cut(t, axes):
    """The same tensors with the neutral sector of the given MPO bonds given as two (where it has two
    states at least): one block more in each, the values moved with their states."""
    def layout(l):
        n, q = list(l.ndims), list(l.qsyms)
        for k in axes:
            z = numpy.flatnonzero((numpy.rint(2 * q[k]) == 0).all(axis=1))[0]
            if n[k][z] > 1:
                n[k] = numpy.insert(n[k], z, 1)
                n[k][z + 1] -= 1
                q[k] = numpy.insert(q[k], z, q[k][z], axis=0)
        return Layout(l.status, q, n)

    states = lambda l: [[int(o) + numpy.arange(int(m)) for o, m in zip(os, ns)]                 # noqa: E731
                        for os, ns in zip(l.secoff, l.ndims)]
    new, vals = [], []
    for i, l in enumerate(t.layouts):
        dense = numpy.zeros(int(numpy.prod(l.shape)))
        dense[l.prjmap(states(l))] = t.op_values(i).numpy()
        new.append(layout(l))
        vals.append(dense[new[-1].prjmap(states(new[-1]))])
    return TensorSet(new, vals, device="cpu"), new[0] is not t.layouts[0]


@pytest.mark.parametrize("tag", ["K4", "K5", "K6"])
def test_a_neutral_sector_given_as_two(tag, monkeypatch):
    """Bit for bit the diagonal of the whole sector: the same states in the same order."""
    patch(monkeypatch)
    cut = 0
    for r in load("kernels_%s.npz" % tag)["records"]:
        sets = [tensorset(r[k], "cpu") for k in ("envL", "envR", "mpo_i", "mpo_j")]
        args = (numpy.asarray(r["qkey"]), [int(v) for v in numpy.atleast_1d(r["opers"])], numpy.atleast_1d(r["hpwts"]))

        def diag(L, R, Wi, Wj):
            return DiagOperator(Workspace(torch.device("cpu")), int(r["key"][2]), layout_of(r["qtmp"]), L, R, Wi, Wj,
                                *args)()
        two = [_cut(t, a) for t, a in zip(sets, ([0], [0], [0, 1], [0, 1]))]
        cut += any(c for _, c in two)
        assert torch.equal(diag(*[t for t, _ in two]), diag(*sets))
    assert cut
