"""Fused orthonormalisation of one Davidson vector (qc_ortho) against the matrix-product form."""
import pytest
import torch

from qcmpodmrg_b200.davidson import _ortho
from qcmpodmrg_b200.engine import LOG


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 4, 5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n", [33, 255, 513, 151553, 300007])
def test_one_vector_against_the_matrix_form(m, n):
    """The basis is orthonormal, so |out| loses digits only as |r| / |r - V^T V r|; sums of n
    products in another order differ by less than sqrt(n) 2^-53 of their terms."""
    gen = torch.Generator().manual_seed(m * 1000003 + n)
    v = torch.linalg.qr(torch.randn(n, m, dtype=torch.float64, generator=gen))[0].T.contiguous()
    r = torch.randn(1, n, dtype=torch.float64, generator=gen)
    k, ref = _ortho(v, r, 1e-12)
    assert k == 1
    loss = float(torch.linalg.norm(r) / torch.linalg.norm(r - (r @ v.T) @ v))
    got, out = _ortho(v.cuda(), r.cuda(), 1e-12)
    out = out.cpu()
    assert got == 1 and out.shape == (1, n)
    tol = 8 * m * n ** 0.5 * 2.0 ** -53 * loss
    assert float((out - ref).abs().max()) <= tol
    assert float((out @ v.T).abs().max()) <= tol and abs(float(torch.linalg.norm(out)) - 1.0) <= tol
    # a vector inside the span has no new direction
    inside = torch.randn(1, m, dtype=torch.float64, generator=gen) @ v
    assert _ortho(v.cuda(), inside.cuda(), 1e-12) == (0, None)


@pytest.mark.gpu
def test_an_empty_basis():
    """Nothing to remove: the vector, normalised."""
    r = torch.tensor([[3.0, 4.0]], dtype=torch.float64)
    k, out = _ortho(torch.zeros(0, 2, dtype=torch.float64, device="cuda"), r.cuda(), 1e-12)
    assert k == 1 and float((out.cpu() - r / 5.0).abs().max()) <= 2.0 ** -52


def test_launches_on_the_device_of_the_vectors(monkeypatch):
    """Stand-ins for vectors of a device that is not the current one: the kernels are launched with
    that device current."""
    from unittest import mock
    from qcmpodmrg_b200 import davidson
    current = ["cuda:0"]

    class Device(object):
        def __init__(self, device):
            self.device = device

        def __enter__(self):
            current.append(self.device)

        def __exit__(self, *a):
            current.pop()

    def vector(rows):
        t = mock.MagicMock(is_cuda=True, dtype=torch.float64, shape=(rows, 9), device="cuda:1")
        t.contiguous.return_value = t
        return t

    seen = []
    lib = mock.MagicMock()
    lib.qc_ortho_work.return_value = 1
    lib.qc_ortho.side_effect = lambda *a: seen.append(current[-1]) or 0
    monkeypatch.setattr(davidson.native, "lib", lambda: lib)
    monkeypatch.setattr(torch, "empty_like", lambda r: r)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d: mock.MagicMock(device=d))
    monkeypatch.setattr(torch.cuda, "device", Device)
    work = mock.MagicMock()
    work.__getitem__.return_value = 1.0
    monkeypatch.setattr(torch, "empty", lambda *a, **k: work)
    before = LOG.launches
    assert _ortho(vector(3), vector(1), 1e-12)[0] == 1
    assert LOG.launches - before == 8           # five passes, the last products, two scalings
    assert seen == ["cuda:1"] and current == ["cuda:0"]
