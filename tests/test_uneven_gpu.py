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
