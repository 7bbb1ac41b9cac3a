"""rbsr in groups of staged rows (B rows of 128 bytes and more) against the FP64
oracle where it can go wrong: each lane layout, rows that fill a stage or
cross several, empty rows, few and many rows per group, matrices smaller than
a block's share, accumulation, 16-bit types, columns outside the matrix.

Bar: 1e-5 of sum|a*b| per element, plus one rounding of a 16-bit output."""
import numpy as np
import pytest
import torch

from gpu_util import dev_csr, oracle64, rounded
from segscan_gb300 import synth

pytestmark = pytest.mark.gpu
U16 = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def shaped(lengths, ncol, seed=0):
    return synth.csr_from_lengths(len(lengths), ncol, np.asarray(lengths, dtype=np.int64), np.random.default_rng(seed))


def check(csr, N, dtype=torch.float32, out_dtype=torch.float32, accumulate=False, what="", **knobs):
    from segscan_gb300 import api
    B = synth.dense(csr.ncol, N, seed=N)
    vals = rounded(csr.values, dtype) if dtype != torch.float32 else csr.values
    C64, absC = oracle64(csr, rounded(B, dtype) if dtype != torch.float32 else B, vals)
    out = torch.full((csr.nrow, N), float("nan"), device="cuda", dtype=out_dtype)
    if accumulate:
        out = torch.from_numpy(synth.dense(csr.nrow, N, seed=N + 1)).cuda().to(out_dtype)
        prev = out.double().cpu().numpy()
        C64, absC = C64 + prev, absC + np.abs(prev)
    got = api.spmm(dev_csr(csr, dtype), torch.from_numpy(B).cuda().to(dtype), "rbsr",
                   knobs=api.make_knobs("rbsr", N, **knobs), out=out, accumulate=accumulate)
    torch.cuda.synchronize()
    err = np.abs(got.double().cpu().numpy() - C64)
    bound = 1e-5 * absC + U16[out_dtype] * np.abs(C64) + 2.0 ** -24
    assert np.all(err <= bound), f"{what}: worst {np.max(err - bound):.3e} over the bound"


SHAPES = {
    "short": [0, 1, 2, 3, 0, 0, 5, 1] * 900,
    "stage": [63, 64, 65, 128, 1, 0, 127, 129] * 40,
    "regular": [20] * 5000,
    "long": [3, 5000, 0, 700, 0, 1, 1500, 64, 2],  # rows above the compensation threshold too
    "one": [17],
    "empties": ([0] * 40 + [9]) * 60,
}


@pytest.mark.parametrize("shape", list(SHAPES))
@pytest.mark.parametrize("accumulate", [False, True])
def test_rows(cuda, shape, accumulate):
    csr = shaped(SHAPES[shape], 9000, seed=3)
    for N in (32, 64, 100, 128, 130, 256):
        check(csr, N, accumulate=accumulate, what=f"{shape} N={N}")


@pytest.mark.parametrize("dtype,out_dtype", [(torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16),
                                             (torch.float16, torch.float16), (torch.float16, torch.float32)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_16bit(cuda, dtype, out_dtype, accumulate):
    csr = shaped(SHAPES["short"] + SHAPES["long"] + SHAPES["stage"], 9000, seed=4)
    for N in (20, 64, 72, 128, 200):
        check(csr, N, dtype, out_dtype, accumulate, f"N={N}")


def test_the_tuple_does_not_change_the_bits(cuda):
    """Each row is summed in order whatever the geometry: the 8-lane layout (N = 32), the 16-lane
    one over the same columns (N = 64) and every tuple give the same bits."""
    from segscan_gb300 import api
    csr = shaped(SHAPES["short"] + SHAPES["long"], 9000, seed=5)
    A = dev_csr(csr)
    B = torch.from_numpy(synth.dense(csr.ncol, 64, seed=6)).cuda()
    wide = api.spmm(A, B, "rbsr")
    for kw in (dict(coarsen_factor=1, tile_factor=3), dict(thread_per_block=64, tile_factor=6)):
        assert torch.equal(wide, api.spmm(A, B, "rbsr", knobs=api.make_knobs("rbsr", 64, **kw)))
    half = api.spmm(A, B[:, :32].contiguous(), "rbsr")
    assert torch.equal(wide[:, :32], half)
    narrow = api.spmm(A, B[:, :4].contiguous(), "rbsr")  # a row per team
    assert torch.equal(wide[:, :4], narrow)


def test_columns_outside_are_skipped(cuda):
    from segscan_gb300 import api
    csr = shaped(SHAPES["stage"], 3000, seed=7)
    A = dev_csr(csr)
    cols, vals = A.indices.clone(), A.values.clone()
    cols[::53] = csr.ncol
    cols[7] = -1
    zeroed = vals.clone()
    zeroed[::53] = 0
    zeroed[7] = 0
    B = torch.from_numpy(synth.dense(csr.ncol, 64, seed=8)).cuda()
    got = api.spmm(api.CsrMatrix(A.nrow, A.ncol, A.indptr, cols, vals), B, "rbsr")
    ref = api.spmm(api.CsrMatrix(A.nrow, A.ncol, A.indptr, A.indices, zeroed), B, "rbsr")
    assert torch.equal(got, ref)
