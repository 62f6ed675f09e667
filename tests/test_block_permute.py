"""Block copies with permuted strides (qc_block_permute) element by element."""
import numpy
import pytest
import torch

from qcmpodmrg_b200.engine import BPERM_DT, op_table, upload
from qcmpodmrg_b200.kernels import block_permute


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 1, 257), (3, 1, 1), (300, 1, 2), (2, 256, 1), (5, 7, 11), (17, 31, 33),
                                  (2, 3, 513), (1, 255, 256)])
@pytest.mark.parametrize("order", [(0, 1, 2), (2, 0, 1), (1, 2, 0)])
def test_copy(dims, order, dtype):
    """Values are copied or rounded to FP32 once: equal bit for bit; padding stays untouched."""
    rng = numpy.random.default_rng(sum(dims) + order[0])
    n = int(numpy.prod(dims))
    src = rng.standard_normal(2 * n + 3)
    # destination: axes in the given order, innermost rows padded by 3
    st = numpy.zeros(3, dtype=numpy.int64)
    st[order[2]] = 1
    st[order[1]] = dims[order[2]] + 3
    st[order[0]] = st[order[1]] * dims[order[1]]
    size = int(st[order[0]]) * dims[order[0]] + 5
    d = numpy.zeros(1, BPERM_DT)
    d["src_off"], d["dst_off"] = 3, 5
    d["d0"], d["d1"], d["d2"] = dims
    d["s0"], d["s1"], d["s2"] = st
    d["op_b"], d["op_e"] = 0, 2
    ops = op_table(numpy.array([0, n]), 0, numpy.array([0, size]), 1.0)
    dst = torch.full((2 * size,), 7.0, dtype=dtype, device="cuda")
    block_permute(upload(d, "cuda"), 1, 2, upload(ops, "cuda"), torch.from_numpy(src).cuda(), dst)
    ref = numpy.full(2 * size, 7.0, dtype=numpy.float64 if dtype == torch.float64 else numpy.float32)
    i = numpy.indices(dims).reshape(3, -1)
    for q in range(2):
        ref[q * size + 5 + st @ i] = src[3 + q * n:3 + (q + 1) * n]
    assert numpy.array_equal(dst.cpu().numpy(), ref)
