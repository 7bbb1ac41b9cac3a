"""The segment tile walk (sequential tuples of up to 2048 elements per run)
against the FP64 oracle where it can go wrong: each lane layout, last tiles
of one element to a whole tile, segments across many tiles and ending on
their boundaries, gaps between ids, ids outside the output, unaligned
operands, the group walk's smaller workspace.

Bar: 1e-5 of sum|x| per element for sums and means, equality for max."""
import numpy as np
import pytest
import torch

import oracle_lib
from gpu_util import rounded

pytestmark = pytest.mark.gpu
REDUCE = {"sum": 0, "max": 1, "mean": 2}


def ids(lengths, gaps):
    """Sorted ids: segment k has lengths[k] elements and gaps[k] empty segments before it."""
    first = np.cumsum(np.asarray(gaps) + 1) - 1
    return np.repeat(first, lengths).astype(np.int32)


def check(index, N, dst_len, reduce, dtype=torch.float32, what="", src=None, out=None, **kw):
    from segscan_gb300 import api
    host = np.random.default_rng(N).uniform(-1, 1, (index.size, N)).astype(np.float32)
    ref, dabs = oracle_lib.segment_coo_f64(rounded(host, dtype) if dtype != torch.float32 else host, index, dst_len,
                                           REDUCE[reduce])
    d = torch.from_numpy(host).cuda().to(dtype)
    if src is not None:
        d = src(d)
    o = torch.full((dst_len, N), float("nan"), device="cuda")
    if out is not None:
        o = out(o)
    got = api.segment(d, torch.from_numpy(index).cuda(), dst_len, reduce, "sr", out=o, **kw)
    torch.cuda.synchronize()
    got = got.double().cpu().numpy()
    if reduce == "max":
        assert np.array_equal(got, ref), what
    else:
        assert np.all(np.abs(got - ref) <= 1e-5 * dabs + 1e-30), what


def mixed(n, seed):
    rng = np.random.default_rng(seed)
    lengths, left = [], n
    while left > 0:
        k = min(left, int(rng.choice([1, 2, 3, 5, 9, 40, 700])))
        lengths.append(k)
        left -= k
    return ids(lengths, rng.choice([0, 0, 0, 1, 2, 45], size=len(lengths)))


WIDTHS = [1, 2, 3, 4, 6, 8, 9, 16, 17, 30, 32, 33, 47, 64, 65, 66, 68, 100, 128, 132]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("reduce", ["sum", "max", "mean"])
def test_lane_layouts(cuda, dtype, reduce):
    index = mixed(20000, 3)
    for N in WIDTHS:
        check(index, N, int(index[-1]) + 4, reduce, dtype, f"N={N}")


@pytest.mark.parametrize("reduce", ["sum", "max", "mean"])
@pytest.mark.parametrize("nnz", [1, 2, 63, 64, 65, 127, 128, 129, 1023, 1024, 1025, 2047, 2049, 4097])
def test_tile_edges(cuda, nnz, reduce):
    for N in (4, 47, 64):
        check(np.arange(nnz, dtype=np.int32), N, nnz + 1, reduce, what=f"singles N={N}")
        check(np.zeros(nnz, dtype=np.int32), N, 3, reduce, what=f"one segment N={N}")
        check(np.repeat(np.arange(-(-nnz // 64)), 64)[:nnz].astype(np.int32), N, nnz, reduce, what=f"64s N={N}")


@pytest.mark.parametrize("reduce", ["sum", "max", "mean"])
@pytest.mark.parametrize("name", ["long", "on_tiles", "wide_gaps"])
def test_segment_shapes(cuda, name, reduce):
    index = {
        "long": ids([3, 30000, 1, 20000, 7], [2, 0, 0, 5, 1]),
        "on_tiles": ids([128] * 40 + [1024] * 3 + [2048, 4096], [0, 3] * 22 + [0]),
        "wide_gaps": ids([5] * 800, [900] * 800),
    }[name]
    for N in (4, 20, 64):
        check(index, N, int(index[-1]) + 300, reduce, what=f"{name} N={N}")


def test_ids_outside_the_output_are_left_out(cuda):
    from segscan_gb300 import api
    index = np.concatenate([[-7, -7, -1], mixed(5000, 9), [9_000_000] * 700, [2**31 - 1]]).astype(np.int32)
    M = int(index[5003 - 1]) + 1
    inside = (index >= 0) & (index < M)
    N = 64
    host = np.random.default_rng(1).uniform(-1, 1, (index.size, N)).astype(np.float32)
    host[~inside] = np.inf
    for reduce in ("sum", "max", "mean"):
        ref, dabs = oracle_lib.segment_coo_f64(np.ascontiguousarray(host[inside]), index[inside], M, REDUCE[reduce])
        out = torch.full((M, N), float("nan"), device="cuda")
        got = api.segment(torch.from_numpy(host).cuda(), torch.from_numpy(index).cuda(), M, reduce, "sr", out=out)
        got = got.double().cpu().numpy()
        assert np.all(np.abs(got - ref) <= 1e-5 * dabs + 1e-30), reduce


def test_accumulate_and_unaligned(cuda):
    from segscan_gb300 import api
    index = mixed(9000, 4)
    M = int(index[-1]) + 2

    def shifted(t):
        buf = torch.zeros(t.numel() + 1, dtype=t.dtype, device="cuda")
        buf[1:] = t.reshape(-1)
        return buf[1:].view(t.shape)

    k = api.make_knobs("ebsr", 64, coarsen_factor=1)  # asks for no vector alignment
    for src, out in ((shifted, None), (None, shifted), (shifted, shifted)):
        check(index, 64, M, "sum", src=src, out=out, knobs=k, what="unaligned")
    for N in (3, 64, 100):
        host = np.random.default_rng(N).uniform(-1, 1, (index.size, N)).astype(np.float32)
        old = np.random.default_rng(N + 1).uniform(-1, 1, (M, N)).astype(np.float32)
        ref, dabs = oracle_lib.segment_coo_f64(host, index, M, 0)
        out = torch.from_numpy(old.copy()).cuda()
        api.segment(torch.from_numpy(host).cuda(), torch.from_numpy(index).cuda(), M, "sum", "sr", out=out,
                    accumulate=True)
        err = np.abs(out.double().cpu().numpy() - (ref + old))
        assert np.all(err <= 1e-5 * (dabs + np.abs(old)) + 1e-30), f"accumulate N={N}"


def test_long_tuples_keep_the_group_walk_and_its_workspace(cuda):
    from segscan_gb300 import api
    index = mixed(60000, 6)
    M, N = int(index[-1]) + 1, 64
    src = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, (index.size, N)).astype(np.float32)).cuda()
    idx = torch.from_numpy(index).cuda()
    ref, dabs = oracle_lib.segment_coo_f64(src.cpu().numpy(), index, M, 0)
    long = api.make_knobs("ebsr", N, thread_nz=256)   # 4096 elements a run: the group walk
    tile = api.make_knobs("ebsr", N, thread_nz=128)   # 2048: the tile walk ...
    small = api.segment_workspace_size(index.size, N, "sr", long)
    assert small < api.segment_workspace_size(index.size, N, "sr", tile)
    chunks = -(-index.size // 2048)  # ... or, in a workspace of the group walk's size, that one
    ws = torch.empty(((chunks * 4 + 255) & ~255) + 2 * chunks * N * 4 + ((2 * chunks * 4 + 255) & ~255) + 512,
                     dtype=torch.uint8, device="cuda")
    for kw in (dict(knobs=long), dict(knobs=tile), dict(knobs=tile, workspace=ws)):
        got = api.segment(src, idx, M, "sum", "sr", **kw).double().cpu().numpy()
        assert np.all(np.abs(got - ref) <= 1e-5 * dabs + 1e-30)
