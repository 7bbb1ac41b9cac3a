"""Work that follows the place in the arrays: rows whose lengths follow their index (rbsr shares out whole
rows), and rows and segments over many tiles.  Such an order costs little against an even one; the times
are the shortest of several, both sides in one process."""
import numpy as np
import pytest
import torch

import test_rb_tile_gpu as rb

pytestmark = pytest.mark.gpu


def shortest(call, n=7):
    call()
    best = float("inf")
    for _ in range(n):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in "ab")
        a.record()
        call()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


# (enough rows that a block's groups take several units each at N = 64)
UNEVEN = {
    "ascending": np.arange(60_000) // 2000,
    "descending": np.arange(60_000)[::-1] // 2000,
    "two kinds": np.where(np.arange(60_000) < 4500, 120, 2),
    "long at the end": np.where(np.arange(130_000) < 129_940, 3, 3000),
    "one full row": np.where(np.arange(160_000) == 90_000, 9_000, 0),
    "full and empty": np.where(np.arange(160_000) % 80_000 < 8_000, 40, 0),
}


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("order", list(UNEVEN))
def test_rows_in_order(cuda, order, accumulate):
    csr = rb.shaped(UNEVEN[order], 9000, seed=5)
    for N in (32, 64, 128, 130):
        rb.check(csr, N, accumulate=accumulate, what=f"{order} N={N}")


def test_time_of_rows_in_order(cuda):
    """One row in ten holds 100 nonzeros: together at the front, or shuffled (482 and 149 us with equal
    numbers of rows per SM)."""
    from segscan_gb300 import api
    M, N = 300_000, 64
    lengths = np.where(np.arange(M) < M // 10, 100, 4)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    times = []
    for L in (lengths, np.random.default_rng(0).permutation(lengths)):
        indptr = torch.from_numpy(np.concatenate([[0], np.cumsum(L)]).astype(np.int32)).cuda()
        cols = torch.randint(0, M, (int(L.sum()),), generator=g, device="cuda", dtype=torch.int32)
        A = api.CsrMatrix(M, M, indptr, cols, torch.rand(cols.numel(), device="cuda"))
        plan, B, C = api.SpmmPlan(A, N, "rbsr"), torch.rand(M, N, device="cuda"), torch.empty(M, N, device="cuda")
        times.append(shortest(lambda: plan.run(B, C)))
    assert times[0] <= 1.6 * times[1], times


def test_time_of_one_long_row(cuda):
    """One row of 4.6 M nonzeros against a hundred of 46 K (767 and 175 us with four heads in flight)."""
    from segscan_gb300 import api
    K, n, N = 200_000, 4_600_000, 64
    cols = torch.randint(0, K, (n,), device="cuda", dtype=torch.int32)
    vals, B = torch.rand(n, device="cuda"), torch.rand(K, N, device="cuda")
    times = []
    for M in (1, 100):
        A = api.CsrMatrix(M, K, torch.arange(0, n + 1, n // M, dtype=torch.int32, device="cuda"), cols, vals)
        plan, C = api.SpmmPlan(A, N, "ebsr"), torch.empty(M, N, device="cuda")
        times.append(shortest(lambda: plan.run(B, C)))
    assert times[0] <= 3.6 * times[1], times


def test_time_of_one_long_segment(cuda):
    """One segment of 30 M elements against 300 of 100 K: what grew with the square of the tiles took
    3287 and 358 us."""
    from segscan_gb300 import api
    n, N = 30_000_000, 4
    src = torch.rand(n, N, device="cuda")
    times = []
    for M in (1, 300):
        index = (torch.arange(n, device="cuda") * M // n).int()
        out = torch.empty(M, N, device="cuda")
        times.append(shortest(lambda: api.segment(src, index, M, "sum", "sr", out=out)))
    assert times[0] <= 6.0 * times[1], times


@pytest.mark.parametrize("reduce", ["sum", "mean", "max"])
@pytest.mark.parametrize("N", [1, 4, 33, 64])
def test_segments_over_many_tiles(cuda, N, reduce):
    """Last tiles one, a few, 31 to 33 and hundreds of tiles away; whole numbers, so every order of the
    additions gives the same sum (below 2^24)."""
    from segscan_gb300 import api
    tile = {1: 2048, 4: 2048, 33: 1024, 64: 1024}[N]  # elements of a full tile, at most
    lengths = [5, tile * 3 + 1, tile * 30, 2, tile * 31 + 7, tile * 32, tile * 33 - 1, 0, tile * 300, 9, tile, tile]
    n, M = sum(lengths), len(lengths)
    index = torch.repeat_interleave(torch.arange(M), torch.tensor(lengths)).int().cuda()
    src = torch.randint(-8, 9, (n, N), generator=torch.Generator().manual_seed(N)).float().cuda()
    got = api.segment(src, index, M, reduce, "sr").double()
    want = torch.zeros(M, N, dtype=torch.float64, device="cuda")
    if reduce == "max":
        want = torch.stack([x.amax(0) if len(x) else want[0] for x in src.double().split(lengths)])
    else:
        want.index_add_(0, index.long(), src.double())
    if reduce == "mean":
        want /= torch.tensor(lengths, device="cuda").clamp(min=1)[:, None]
        assert torch.all((got - want).abs() <= 2.0 ** -24 * want.abs())  # one division, rounded
    else:
        assert torch.equal(got, want)
