"""Matrices whose arrays go on after the last row (indptr[nrow] < nnz, columns -1): COO -> CSR makes them of
edges with rows outside the matrix, the transpose of columns outside it.  Every row of C is written and
right, above and below one wave of tiles, whatever the scratch held before (1e-5 of sum|a*b|)."""
import numpy as np
import pytest
import torch

import oracle_lib

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1, 255])
def scratch(request, monkeypatch):
    from segscan_gb300 import api
    monkeypatch.setattr(api, "_workspace",
                        lambda n, device: torch.full((n + 256,), request.param, dtype=torch.uint8, device=device))
    return request.param


def dropping(nnz, nrow, dropped, seed=2):
    """rows, cols (int32) with `dropped` rows outside, the last 40 rows of the matrix and some others empty."""
    rng = np.random.default_rng(seed)
    rows = rng.integers(0, nrow - 40, size=nnz)
    rows[rows % 5 == 2] += 1
    rows[rng.permutation(nnz)[:dropped]] = nrow + 3
    return rows.astype(np.int32), rng.integers(0, nrow, size=nnz).astype(np.int32)


def expect(rows, cols, vals, nrow, B):
    keep = np.flatnonzero(rows < nrow)
    order = keep[np.argsort(rows[keep], kind="stable")]
    indptr = np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=nrow))]).astype(np.int32)
    return oracle_lib.spmm_f64(indptr, cols[order], vals[order], B, threads=8)


@pytest.mark.parametrize("N,nnz", [(4, 9000), (4, 1_500_000), (64, 9000), (64, 900_000), (33, 900_000)])
@pytest.mark.parametrize("dropped", [1, 700, 6000])
def test_spmm(cuda, scratch, N, nnz, dropped):
    from segscan_gb300 import api
    nrow = 5000
    rows, cols = dropping(nnz, nrow, dropped)
    vals = np.random.default_rng(1).uniform(-1, 1, nnz).astype(np.float32)
    A, _ = api.coo_to_csr(nrow, torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda(), ncol=nrow,
                          values=torch.from_numpy(vals).cuda())
    B = np.random.default_rng(7).uniform(-1, 1, (nrow, N)).astype(np.float32)
    got = api.spmm(A, torch.from_numpy(B).cuda(), "ebsr").double().cpu().numpy()
    want, terms = expect(rows, cols, vals, nrow, B)
    assert np.all(np.abs(got - want) <= 1e-5 * terms + 1e-30)


@pytest.mark.parametrize("N", [4, 64])
def test_gradient_of_B(cuda, scratch, N):
    """dB = A^T dC where A has columns outside: A^T's arrays go on after its last row."""
    from segscan_gb300 import api, autograd
    nnz, n = 1_500_000, 5000
    cols, rows = dropping(nnz, n, 6000)
    rows = np.sort(rows)
    indptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    vals = np.random.default_rng(1).uniform(-1, 1, nnz).astype(np.float32)
    A = api.CsrMatrix(n, n, torch.from_numpy(indptr).cuda(), torch.from_numpy(cols).cuda(), torch.from_numpy(vals).cuda())
    B = torch.zeros(n, N, device="cuda", requires_grad=True)
    dC = np.random.default_rng(7).uniform(-1, 1, (n, N)).astype(np.float32)
    autograd.spmm(A, A.values, B).backward(torch.from_numpy(dC).cuda())
    want, terms = expect(cols, rows, vals, n, dC)
    assert np.all(np.abs(B.grad.double().cpu().numpy() - want) <= 1e-5 * terms + 1e-30)


@pytest.mark.parametrize("N", [4, 64, 100, 128, 256])
@pytest.mark.parametrize("nrow,nnz,dropped", [(5000, 9000, 700), (41, 300, 299), (50, 50, 50), (5000, 300_000, 6000)])
def test_gradient_of_the_values(cuda, N, nrow, nnz, dropped):
    """SDDMM: 0 for entries that follow the last row, whose columns are -1."""
    from segscan_gb300 import api
    rows, cols = dropping(nnz, nrow, dropped)
    A, perm = api.coo_to_csr(nrow, torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda(), ncol=nrow)
    rng = np.random.default_rng(3)
    dC, B = (rng.uniform(-1, 1, (nrow, N)).astype(np.float32) for _ in "ab")
    got = api.sddmm(A, torch.from_numpy(dC).cuda(), torch.from_numpy(B).cuda()).double().cpu().numpy()
    kept = perm.cpu().numpy()[:nnz - dropped]
    want = np.einsum("ij,ij->i", dC[rows[kept]].astype(np.float64), B[cols[kept]])
    terms = np.einsum("ij,ij->i", np.abs(dC[rows[kept]]).astype(np.float64), np.abs(B[cols[kept]]))
    assert np.all(np.abs(got[:nnz - dropped] - want) <= 1e-5 * terms + 1e-30)
    assert np.all(got[nnz - dropped:] == 0)


@pytest.mark.parametrize("strategy", ["ebpr", "rbpr", "rbsr"])
@pytest.mark.parametrize("N,nnz,dropped", [(4, 9000, 700), (33, 9000, 6000), (64, 300_000, 1), (64, 300_000, 9000)])
def test_other_strategies(cuda, scratch, strategy, N, nnz, dropped):
    """(the last row has nonzeros here, and chunks of dropped entries follow its own)"""
    from segscan_gb300 import api
    nrow = 5000
    rows, cols = dropping(nnz, nrow, dropped)
    rows[np.flatnonzero(rows < nrow)[:7]] = nrow - 1
    vals = np.random.default_rng(1).uniform(-1, 1, nnz).astype(np.float32)
    A, _ = api.coo_to_csr(nrow, torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda(), ncol=nrow,
                          values=torch.from_numpy(vals).cuda())
    B = np.random.default_rng(7).uniform(-1, 1, (nrow, N)).astype(np.float32)
    got = api.spmm(A, torch.from_numpy(B).cuda(), strategy).double().cpu().numpy()
    want, terms = expect(rows, cols, vals, nrow, B)
    assert np.all(np.abs(got - want) <= 1e-5 * terms + 1e-30)


@pytest.mark.parametrize("N", [4, 33, 64])
@pytest.mark.parametrize("strategy", ["rbsr", "ebsr"])
def test_batched(cuda, strategy, N):
    """Trailing empty rows are written too; the last matrix has dropped edges only."""
    from segscan_gb300 import api, autotune
    from segscan_gb300.batched import BatchedSpMM
    mats, Bs, wants = [], [], []
    for i, (nrow, nnz, dropped) in enumerate([(5000, 9000, 700), (60, 300, 1), (900, 40_000, 9000), (50, 70, 70)]):
        rows, cols = dropping(nnz, nrow, dropped, seed=i)
        vals = np.random.default_rng(1).uniform(-1, 1, nnz).astype(np.float32)
        B = np.random.default_rng(7).uniform(-1, 1, (nrow, N)).astype(np.float32)
        mats.append(api.coo_to_csr(nrow, torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda(), ncol=nrow,
                                   values=torch.from_numpy(vals).cuda())[0])
        Bs.append(torch.from_numpy(B).cuda())
        wants.append(expect(rows, cols, vals, nrow, B))
    outs = BatchedSpMM(mats, Bs, knobs=autotune.batch_knobs(mats, N), strategies=[strategy] * len(mats)).run()
    for got, (want, terms) in zip(outs, wants):
        assert np.all(np.abs(got.double().cpu().numpy() - want) <= 1e-5 * terms + 1e-30)


@pytest.mark.parametrize("N,nnz,dropped", [(4, 9000, 700), (33, 9000, 6000), (64, 300_000, 1), (64, 300_000, 20_000)])
def test_group_walk(cuda, scratch, N, nnz, dropped):
    """ebsr with runs above 2048 nonzeros: chunks that hold the last row and dropped entries, or these alone."""
    from segscan_gb300 import api
    nrow = 5000
    knobs = api.make_knobs("ebsr", N, thread_nz=4096)
    for last in (0, 7):
        rows, cols = dropping(nnz, nrow, dropped)
        rows[np.flatnonzero(rows < nrow)[:last]] = nrow - 1
        vals = np.random.default_rng(1).uniform(-1, 1, nnz).astype(np.float32)
        A, _ = api.coo_to_csr(nrow, torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda(), ncol=nrow,
                              values=torch.from_numpy(vals).cuda())
        B = np.random.default_rng(7).uniform(-1, 1, (nrow, N)).astype(np.float32)
        got = api.spmm(A, torch.from_numpy(B).cuda(), "ebsr", knobs=knobs).double().cpu().numpy()
        want, terms = expect(rows, cols, vals, nrow, B)
        assert np.all(np.abs(got - want) <= 1e-5 * terms + 1e-30)


@pytest.mark.parametrize("N", [4, 64, 128])
def test_both_gradients(cuda, N):
    """One walk over A^T gives both; nonzeros that A^T does not hold get 0."""
    from segscan_gb300 import api, autograd
    nnz, n, dropped = 60_000, 5000, 6000
    cols, rows = dropping(nnz, n, dropped)
    rows = np.sort(rows)
    indptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    vals = np.random.default_rng(1).uniform(-1, 1, nnz).astype(np.float32)
    rng = np.random.default_rng(3)
    dC, Bh = (rng.uniform(-1, 1, (n, N)).astype(np.float32) for _ in "ab")
    A = api.CsrMatrix(n, n, torch.from_numpy(indptr).cuda(), torch.from_numpy(cols).cuda(), None)
    v = torch.from_numpy(vals).cuda().requires_grad_(True)
    B = torch.from_numpy(Bh).cuda().requires_grad_(True)
    autograd.spmm(A, v, B).backward(torch.from_numpy(dC).cuda())
    kept = cols < n
    want = np.where(kept, np.einsum("ij,ij->i", dC[rows].astype(np.float64), Bh[np.where(kept, cols, 0)]), 0)
    terms = np.einsum("ij,ij->i", np.abs(dC[rows]).astype(np.float64), np.abs(Bh[np.where(kept, cols, 0)]))
    assert np.all(np.abs(v.grad.double().cpu().numpy() - want) <= 1e-5 * terms)
    want, terms = expect(cols, rows, vals, n, dC)
    assert np.all(np.abs(B.grad.double().cpu().numpy() - want) <= 1e-5 * terms + 1e-30)
