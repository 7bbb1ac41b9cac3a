"""Accumulating at widths that leave lanes of a group without a column: each element is added to once.
Whole numbers, so every result is exact."""
import pytest
import torch

from gpu_util import dev_csr
from segscan_gb300 import synth

pytestmark = pytest.mark.gpu
WIDTHS = [3, 9, 33, 47, 63, 66, 100, 132]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("strategy", ["ebsr", "rbsr"])
@pytest.mark.parametrize("mean", [0.3, 6.0])  # the first is hypersparse: zeroed, then accumulated
def test_spmm(cuda, strategy, mean, dtype):
    from segscan_gb300 import api
    csr = synth.poisson(20_000, 3000, mean, seed=4)
    A = dev_csr(csr, values=False)
    A = A.with_values(torch.ones(A.nnz, device="cuda", dtype=dtype))
    count = (A.indptr[1:] - A.indptr[:-1]).float()
    for N in WIDTHS:
        B = torch.ones(3000, N, device="cuda", dtype=dtype)
        assert torch.equal(api.spmm(A, B, strategy), count[:, None].expand(-1, N))
        C = torch.ones(csr.nrow, N, device="cuda")
        for k in range(1, 5):
            api.spmm(A, B, strategy, out=C, accumulate=True)
            assert torch.equal(C, (k * count + 1)[:, None].expand(-1, N)), f"N={N} call {k}"


@pytest.mark.parametrize("rows", [9000, 400_000])
def test_segment(cuda, rows):
    from segscan_gb300 import api
    index = (torch.arange(60_000, device="cuda") // 7).int()
    count = torch.bincount(index, minlength=rows).float()
    for N in WIDTHS:
        src = torch.ones(index.numel(), N, device="cuda")
        assert torch.equal(api.segment(src, index, rows, "sum", "sr"), count[:, None].expand(-1, N))
        C = torch.ones(rows, N, device="cuda")
        for k in range(1, 5):
            api.segment(src, index, rows, "sum", "sr", out=C, accumulate=True)
            assert torch.equal(C, (k * count + 1)[:, None].expand(-1, N)), f"N={N} call {k}"
