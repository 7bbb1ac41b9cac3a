"""Infinities in the terms of a sum: a row (or segment) with one is infinite, whatever piece, tile or
chunk of the walk holds it, one whose partial sums overflow too, and one with both signs is NaN; every
other row keeps its value (1e-5 of sum|terms|)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# short rows, rows across pieces and tiles (8 to 128 nonzeros, 128 to 2048), one above the compensation
# threshold of 1024, one of every length in between
LENGTHS = [3, 10, 37, 5, 300, 1500, 9, 64, 0, 65, 700, 1, 20, 130, 2]
SPMM = [("ebsr", {}), ("ebsr", dict(thread_nz=256)), ("rbsr", {}), ("rbpr", {}), ("ebpr", {})]
KINDS = {"inf": (np.inf, 0.0), "neg": (-np.inf, 0.0), "overflow": (3e38, 3e38), "both": (np.inf, -np.inf)}


def placed(n, N, first, kind):
    """Terms in (0, 1): column j has the kind's values at elements first + j and first + j + 1."""
    x = np.random.default_rng(5).uniform(0.1, 1, (n, N)).astype(np.float32)
    rows = np.repeat(np.arange(len(LENGTHS)), LENGTHS)
    want = np.zeros((len(LENGTHS), N))
    np.add.at(want, rows, x.astype(np.float64))
    with np.errstate(invalid="ignore"):
        for j in range(N):
            p = min(first + j, n - 2)
            for q, v in zip((p, p + 1), KINDS[kind]):
                if v != 0.0:
                    want[rows[q], j] += v - float(x[q, j])
                    x[q, j] = v
        return x, np.where(np.abs(want) > 3.4e38, np.sign(want) * np.inf, want)


def check(got, want, what):
    got = got.double().cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(want)), f"{what}: NaN"
    assert np.array_equal(np.isinf(got), np.isinf(want)), f"{what}: Inf"
    inf = np.isinf(want)
    assert np.array_equal(np.sign(got[inf]), np.sign(want[inf])), f"{what}: sign"
    fin = np.isfinite(want)
    assert np.all(np.abs(got[fin] - want[fin]) <= 1e-5 * np.abs(want[fin])), what


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("strategy,kw", SPMM)
@pytest.mark.parametrize("N", [4, 33, 64])
def test_spmm(cuda, N, strategy, kw, kind):
    from segscan_gb300 import api
    n = sum(LENGTHS)
    indptr = np.concatenate([[0], np.cumsum(LENGTHS)]).astype(np.int32)
    A = api.CsrMatrix(len(LENGTHS), n, torch.from_numpy(indptr).cuda(), torch.arange(n, dtype=torch.int32, device="cuda"),
                      torch.ones(n, device="cuda"))
    for first in list(range(0, 420, max(N, 24))) + list(range(1000, n, 170)):
        B, want = placed(n, N, first, kind)
        got = api.spmm(A, torch.from_numpy(B).cuda(), strategy, knobs=api.make_knobs(strategy, N, **kw) if kw else None)
        check(got, want, f"N={N} first={first}")


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("reduce", ["sum", "mean"])
@pytest.mark.parametrize("strategy", ["sr", "pr"])
@pytest.mark.parametrize("N", [4, 33, 64])
def test_segment(cuda, N, strategy, reduce, kind):
    from segscan_gb300 import api
    n, M = sum(LENGTHS), len(LENGTHS)
    index = torch.from_numpy(np.repeat(np.arange(M), LENGTHS).astype(np.int32)).cuda()
    for first in list(range(0, 420, max(N, 24))) + list(range(1000, n, 170)):
        x, want = placed(n, N, first, kind)
        if reduce == "mean":
            want = want / np.maximum(LENGTHS, 1)[:, None]
        check(api.segment(torch.from_numpy(x).cuda(), index, M, reduce, strategy), want, f"N={N} first={first}")


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_rbsr_leaves_out_the_value_of_a_column_outside(cuda, value):
    """A nonzero whose column is not in the matrix adds nothing, whatever its value."""
    from segscan_gb300 import api
    lengths = [3, 10, 70, 5, 1500]
    n = sum(lengths)
    indptr = torch.from_numpy(np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)).cuda()
    cols = torch.arange(n, dtype=torch.int32, device="cuda")
    vals = torch.ones(n, device="cuda")
    for N in (4, 33, 64):
        B = torch.rand(n, N, device="cuda")
        ref = api.spmm(api.CsrMatrix(len(lengths), n, indptr, cols, vals.index_fill(0, cols[::9].long(), 0)), B, "rbsr")
        bad, v = cols.clone(), vals.clone()
        bad[::18], bad[9::18], v[::9] = n, -1, value
        got = api.spmm(api.CsrMatrix(len(lengths), n, indptr, bad, v), B, "rbsr")
        assert torch.all((got - ref).abs() <= 1e-5 * ref.abs()), f"N={N}"


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_ebsr_leaves_out_the_value_of_a_column_outside(cuda, value):
    """The same in the tile walk, below and above one wave of tiles."""
    from segscan_gb300 import api
    for lengths in ([3, 10, 70, 5, 1500], [7] * 200_000):
        n = sum(lengths)
        indptr = torch.from_numpy(np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)).cuda()
        cols = torch.arange(n, dtype=torch.int32, device="cuda") % 5000
        vals = torch.ones(n, device="cuda")
        at = torch.arange(0, n, 9, device="cuda")
        bad, v = cols.clone(), vals.clone()
        bad[::18], bad[9::18], v[::9] = 5000, -1, value
        for N in (1, 4, 33, 64):
            B = torch.rand(5000, N, device="cuda")
            ref = api.spmm(api.CsrMatrix(len(lengths), 5000, indptr, cols, vals.index_fill(0, at, 0)), B, "ebsr")
            got = api.spmm(api.CsrMatrix(len(lengths), 5000, indptr, bad, v), B, "ebsr")
            assert torch.all((got - ref).abs() <= 1e-5 * ref.abs()), f"N={N} rows={len(lengths)}"


@pytest.mark.parametrize("value", [1.0, np.inf, np.nan])
@pytest.mark.parametrize("strategy,kw", SPMM + [("ebsr", dict(thread_nz=4096))])
def test_columns_outside_add_nothing(cuda, strategy, kw, value):
    """Whatever the value there and in any row of B that no other nonzero names (rows 0 and K - 1)."""
    from segscan_gb300 import api
    n = sum(LENGTHS)
    indptr = torch.from_numpy(np.concatenate([[0], np.cumsum(LENGTHS)]).astype(np.int32)).cuda()
    cols = 1 + torch.arange(n, dtype=torch.int32, device="cuda")
    vals = torch.ones(n, device="cuda")
    bad, v = cols.clone(), vals.clone()
    bad[::18], bad[9::18], v[::9] = n + 2, -1, value
    at = torch.arange(0, n, 9, device="cuda")
    for N in (4, 33, 64):
        knobs = api.make_knobs(strategy, N, **kw) if kw else None
        B = torch.rand(n + 2, N, device="cuda")
        ref = api.spmm(api.CsrMatrix(len(LENGTHS), n + 2, indptr, cols, vals.index_fill(0, at, 0)), B, strategy, knobs=knobs)
        B[0], B[n + 1] = np.inf, np.nan
        got = api.spmm(api.CsrMatrix(len(LENGTHS), n + 2, indptr, bad, v), B, strategy, knobs=knobs)
        assert torch.all((got - ref).abs() <= 1e-5 * ref.abs()), f"N={N}"
