"""The tile walk (ebsr tuples of up to 2048 nonzeros per run) against the FP64
oracle and against the group walk, at the places where it can go wrong: each
lane layout, last tiles of one nonzero to a whole tile, rows across several
tiles, runs of empty rows, pointers that allow no wide vector, accumulation,
16-bit storage and output, columns outside the matrix.

FP32 bar: 1e-5 of sum|a*b| per element; a 16-bit output adds its one
rounding (2^-8 BF16, 2^-11 FP16)."""
import numpy as np
import pytest
import torch

from gpu_util import dev_csr, oracle64, rounded
from segscan_gb300 import synth

pytestmark = pytest.mark.gpu
U16 = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def shaped(lengths, ncol, seed=0):
    return synth.csr_from_lengths(len(lengths), ncol, np.asarray(lengths, dtype=np.int64), np.random.default_rng(seed))


def mixed(nnz, seed=3):
    """Short, empty and long rows (one above the compensation threshold) with exactly nnz nonzeros
    before duplicate columns are dropped."""
    rng = np.random.default_rng(seed)
    lengths, left = [], nnz
    pool = [1, 2, 3, 0, 0, 7, 40, 0, 0, 0, 0, 0, 300]
    if nnz > 6000:
        lengths += [5, 5000, 0]
        left -= 5005
    while left > 0:
        n = min(left, int(rng.choice(pool)))
        lengths.append(n)
        left -= n
    return lengths + [0, 0, 0]


def check(csr, B, A, Bd, dtype, out_dtype, what, C0=None, **kw):
    from segscan_gb300 import api
    vals = rounded(csr.values, dtype) if dtype != torch.float32 else csr.values
    C64, absC = oracle64(csr, rounded(B, dtype) if dtype != torch.float32 else B, vals)
    out = None
    if C0 is not None:
        out = torch.from_numpy(C0.copy()).cuda().to(out_dtype)
        prev = out.double().cpu().numpy()
        C64, absC = C64 + prev, absC + np.abs(prev)
    got = api.spmm(A, Bd, "ebsr", out=out, out_dtype=out_dtype, accumulate=C0 is not None, **kw)
    torch.cuda.synchronize()
    err = np.abs(got.double().cpu().numpy() - C64)
    bound = 1e-5 * absC + U16[out_dtype] * np.abs(C64) + 2.0 ** -24
    assert np.all(err <= bound), f"{what}: worst {np.max(err - bound):.3e} over the bound"


# one width per lane layout: (16-byte vectors) 4, 8, 16, 32, 64 and two phases;
# (8 bytes) 2 .. 34, 66; (one element) 1 .. 17, 33, 47, 63, 65
WIDTHS = [1, 2, 3, 4, 5, 6, 8, 9, 15, 16, 17, 22, 32, 33, 34, 47, 63, 64, 65, 66, 100, 128]


@pytest.mark.parametrize("dtype,out_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32),
                                             (torch.float16, torch.float16), (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_lane_layouts(cuda, dtype, out_dtype, accumulate):
    csr = shaped(mixed(20000), 3000)
    A = dev_csr(csr, dtype)
    for N in WIDTHS:
        B = synth.dense(csr.ncol, N, seed=N)
        C0 = synth.dense(csr.nrow, N, seed=N + 1) if accumulate else None
        check(csr, B, A, torch.from_numpy(B).cuda().to(dtype), dtype, out_dtype, f"N={N}", C0)


@pytest.mark.parametrize("N", [4, 16, 47, 64])
@pytest.mark.parametrize("nnz", [1, 3, 8, 127, 128, 129, 511, 512, 513, 2047, 2048, 2049, 4096, 9001])
def test_tile_edges(cuda, N, nnz):
    lengths = np.ones(nnz, dtype=np.int64)  # one nonzero a row: no duplicates, exactly nnz
    csr = shaped(lengths, 500, seed=nnz)
    assert csr.nnz == nnz
    B = synth.dense(csr.ncol, N, seed=7)
    check(csr, B, dev_csr(csr), torch.from_numpy(B).cuda(), torch.float32, torch.float32, f"nnz={nnz} N={N}")


@pytest.mark.parametrize("N", [4, 30, 64])
@pytest.mark.parametrize("name", ["one_row", "two_long", "long_then_empty", "ends_on_tiles", "mostly_empty"])
def test_row_shapes(cuda, N, name):
    lengths = {
        "one_row": [30000],
        "two_long": [9000, 0, 0, 12000],
        "long_then_empty": [4096] + [0] * 700 + [2, 0, 1],
        "ends_on_tiles": [128] * 64 + [1024, 0, 1024, 2048, 0],
        "mostly_empty": ([0] * 50 + [60]) * 200,
    }[name]
    csr = shaped(lengths, 40000, seed=1)
    B = synth.dense(csr.ncol, N, seed=2)
    A, Bd = dev_csr(csr), torch.from_numpy(B).cuda()
    check(csr, B, A, Bd, torch.float32, torch.float32, f"{name} N={N}")
    check(csr, B, A, Bd, torch.float32, torch.float32, f"{name} N={N} accumulating",
          synth.dense(csr.nrow, N, seed=3))


def test_unaligned_operands(cuda):
    """B, C, columns and values that start between 16-byte words."""
    from segscan_gb300 import api
    csr = shaped(mixed(9000, seed=5), 2000)
    N = 64
    B = synth.dense(csr.ncol, N, seed=4)
    knobs = api.make_knobs("ebsr", N, coarsen_factor=1)  # asks for no vector alignment

    def shifted(t):
        buf = torch.zeros(t.numel() + 1, dtype=t.dtype, device="cuda")
        buf[1:] = t.reshape(-1)
        return buf[1:].view(t.shape)

    A = dev_csr(csr)
    A2 = api.CsrMatrix(A.nrow, A.ncol, A.indptr, shifted(A.indices), shifted(A.values))
    C64, absC = oracle64(csr, B)
    for a, b in ((A2, False), (A, True), (A2, True)):
        Bd = torch.from_numpy(B).cuda()
        out = shifted(torch.full((csr.nrow, N), float("nan"), device="cuda"))
        got = api.spmm(a, shifted(Bd) if b else Bd, "ebsr", knobs=knobs, out=out)
        err = np.abs(got.double().cpu().numpy() - C64)
        assert np.all(err <= 1e-5 * absC + 1e-30)


def test_columns_outside_are_skipped_like_the_group_walk(cuda):
    from segscan_gb300 import api
    csr = shaped(mixed(7000, seed=6), 1000)
    N = 64
    A = dev_csr(csr)
    bad = A.indices.clone()
    bad[::97] = csr.ncol  # one past the last column
    bad[5] = -1
    A = api.CsrMatrix(A.nrow, A.ncol, A.indptr, bad, A.values)
    Bd = torch.from_numpy(synth.dense(csr.ncol, N, seed=8)).cuda()
    Bd[0] = float("inf")  # a skipped nonzero must not touch any row of B
    tile = api.spmm(A, Bd, "ebsr", knobs=api.make_knobs("ebsr", N))
    walk = api.spmm(A, Bd, "ebsr", knobs=api.make_knobs("ebsr", N, thread_nz=129))  # 129 * 16 > 2048: group walk
    both = torch.isfinite(walk)
    assert torch.equal(both, torch.isfinite(tile))
    scale = api.spmm(api.CsrMatrix(A.nrow, A.ncol, A.indptr, A.indices, A.values.abs()), Bd.abs(), "ebsr")
    assert torch.all((tile - walk).abs()[both] <= 1e-5 * scale[both] + 1e-30)


def test_scratch_of_the_group_walk_is_still_accepted(cuda):
    """A workspace as small as the group walk's (what callers of older versions hold) runs that walk."""
    from segscan_gb300 import api
    csr = synth.powerlaw(40000, 40000, 2.1, 1, 4000, seed=2)
    N = 64
    A = dev_csr(csr)
    Bd = torch.from_numpy(synth.dense(csr.ncol, N, seed=1)).cuda()
    knobs = api.make_knobs("ebsr", N, thread_nz=128)  # 2048 nonzeros a run: the tile walk's by default
    big = api.spmm_workspace_size(A, N, "ebsr", knobs)
    chunks = -(-csr.nnz // 2048)
    walk = ((chunks * 4 + 255) & ~255) + 2 * chunks * N * 4
    assert walk < big
    ref = api.spmm(A, Bd, "ebsr", knobs=knobs)
    small = torch.empty(walk + 256, dtype=torch.uint8, device="cuda")
    small = small[(-small.data_ptr()) % 256:][:walk]
    got = api.spmm(A, Bd, "ebsr", knobs=knobs, workspace=small)
    C64, absC = oracle64(csr, Bd.cpu().numpy())
    for C in (ref, got):
        assert np.all(np.abs(C.double().cpu().numpy() - C64) <= 1e-5 * absC + 1e-30)


@pytest.mark.parametrize("N,nnz", [(4, 1_100_000), (4, 1_400_000), (256, 140_000), (256, 170_000)])
def test_rows_searched_and_listed(cuda, N, nnz):
    """On both sides of one wave of blocks: below it each block searches its rows, above it a kernel lists them."""
    csr = shaped(mixed(nnz), 6000)
    B = synth.dense(csr.ncol, N, seed=N)
    check(csr, B, dev_csr(csr, torch.float32), torch.from_numpy(B).cuda(), torch.float32, torch.float32, f"nnz={nnz}")
