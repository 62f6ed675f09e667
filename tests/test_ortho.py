"""Fused orthonormalisation of one Davidson vector (qc_ortho) against the matrix-product form."""
import pytest
import torch

from qcmpodmrg_b200.davidson import _ortho


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
