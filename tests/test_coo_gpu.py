"""COO -> CSR (the two-level stable sort) bit for bit against a stable argsort
at the sizes where it can go wrong: tiles and chunks and their neighbours,
buckets longer than a chunk, one key per bucket, as many buckets as there may
be, rows outside the matrix, every value type."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def check(nrow, rows, dtype=torch.float32, seed=0):
    from segscan_gb300 import api
    rng = np.random.default_rng(seed)
    nnz = rows.size
    rows = rows.astype(np.int32)
    cols = rng.integers(0, 1 << 30, size=nnz).astype(np.int32)
    vals = torch.from_numpy(rng.standard_normal(nnz).astype(np.float32)).to(dtype)
    A, perm = api.coo_to_csr(nrow, torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda(), ncol=1 << 30,
                             values=vals.cuda())
    B, perm2 = api.coo_to_csr(nrow, torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda(), ncol=1 << 30)
    torch.cuda.synchronize()
    valid = (rows >= 0) & (rows < nrow)
    order = np.nonzero(valid)[0][np.argsort(rows[valid], kind="stable")].astype(np.int32)
    m = order.size
    indptr = np.concatenate([[0], np.cumsum(np.bincount(rows[valid], minlength=nrow))]).astype(np.int32)
    assert np.array_equal(A.indptr.cpu().numpy(), indptr)
    assert np.array_equal(perm.cpu().numpy()[:m], order)
    assert np.all(perm.cpu().numpy()[m:] == -1)
    assert np.array_equal(A.indices.cpu().numpy()[:m], cols[order])
    assert torch.equal(A.values.cpu()[:m], vals[torch.from_numpy(order.astype(np.int64))])
    assert torch.equal(perm, perm2) and torch.equal(A.indptr, B.indptr) and torch.equal(A.indices, B.indices)


@pytest.mark.parametrize("nnz", [1, 31, 33, 511, 512, 4095, 4096, 4097, 8191, 8192, 8193, 40000])
@pytest.mark.parametrize("nrow", [1, 2, 5, 1000, 5000])
def test_sizes(cuda, nnz, nrow):
    rng = np.random.default_rng(nnz * 7 + nrow)
    check(nrow, rng.integers(0, nrow, size=nnz))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", ["sorted", "reversed", "one_row", "two_hubs", "out_of_range", "all_out", "many_rows"])
def test_orders(cuda, case, dtype):
    rng = np.random.default_rng(11)
    nrow, nnz = 6000, 90000
    rows = rng.integers(0, nrow, size=nnz)
    if case == "sorted":
        rows = np.sort(rows)
    elif case == "reversed":
        rows = np.sort(rows)[::-1].copy()
    elif case == "one_row":
        rows[:] = 4321
    elif case == "two_hubs":
        rows[::2] = 17
        rows[1::5] = 18
    elif case == "out_of_range":
        rows[::3] = nrow
        rows[::7] = -5
    elif case == "all_out":
        rows[:] = nrow + 1
    elif case == "many_rows":  # 4096 rows per bucket, and more buckets than a block has threads
        nrow = 3_000_000
        rows = rng.integers(0, nrow, size=nnz)
    check(nrow, rows, dtype)


def test_many_buckets(cuda):
    """More buckets than threads, two blocks' count tables past one SM, and hubs among short rows."""
    rng = np.random.default_rng(5)
    nrow, nnz = 2_500_000, 9_000_000
    rows = rng.integers(0, nrow, size=nnz)
    rows[rng.random(nnz) < 0.02] = 1_234_567
    check(nrow, rows)


def test_old_workspace_is_still_accepted(cuda):
    """A workspace of the one-level sort's size (smaller) runs that sort, with the same result."""
    import ctypes

    from segscan_gb300 import _lib
    rng = np.random.default_rng(2)
    nrow, nnz = 4000, 50000
    rows = torch.from_numpy(rng.integers(0, nrow, size=nnz).astype(np.int32)).cuda()
    cols = torch.from_numpy(rng.integers(0, nrow, size=nnz).astype(np.int32)).cuda()
    n = ctypes.c_size_t()
    _lib.call("ss_coo_to_csr_workspace_size", nrow, nnz, ctypes.byref(n))
    up = lambda x: (x + 255) & ~255
    old = 2 * up((nrow + 1) * 4) + up(nrow * 4) + 2 * 256 + up(4096 * 4) + up(nnz * 4)
    assert old < n.value
    got = []
    for size in (int(n.value), old):
        ws = torch.empty(size + 256, dtype=torch.uint8, device="cuda")
        out = [torch.full((k,), -7, dtype=torch.int32, device="cuda") for k in (nrow + 1, nnz, nnz)]
        p = ws.data_ptr() + (-ws.data_ptr()) % 256
        _lib.call("ss_coo_to_csr", nrow, nnz, rows.data_ptr(), cols.data_ptr(), *[t.data_ptr() for t in out], p, size,
                  torch.cuda.current_stream().cuda_stream)
        got.append(out)
    torch.cuda.synchronize()
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("nrow,nnz", [(300, 5000), (6000, 90000), (5, 40000)])
def test_values_of_rows_outside_are_zero(cuda, nrow, nnz, dtype):
    """Past indptr[nrow]: -1 in the columns and the permutation, zero in the values, as the one-level sort leaves them."""
    from segscan_gb300 import api
    rng = np.random.default_rng(4)
    rows = rng.integers(-2, nrow + 2, size=nnz).astype(np.int32)
    A, perm = api.coo_to_csr(nrow, torch.from_numpy(rows).cuda(), torch.zeros(nnz, dtype=torch.int32, device="cuda"),
                             ncol=1, values=torch.ones(nnz, device="cuda", dtype=dtype))
    m = int(((rows >= 0) & (rows < nrow)).sum())
    assert m < nnz and int(A.indptr[-1]) == m
    assert torch.all(A.values[:m] == 1) and torch.all(A.values[m:] == 0)
    assert torch.all(A.indices[m:] == -1) and torch.all(perm[m:] == -1)
