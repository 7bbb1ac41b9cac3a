"""What this library is used for, as cases that can be timed: SpMM with each
strategy, segment reductions, training steps, the device transpose and COO
conversion, and the batched launch, each through the entry point a program
calls, on the synthetic matrices the benchmark configurations name.

A case is a dict of plain values; ``prepare`` makes on the GPU what a program
has in hand before the call and ``run`` is one pass.  Matrices follow the
row-length laws of ``segscan_gb300.synth`` (made on the GPU here, since they
are made many times): columns sorted and distinct inside a row, values and
dense operands U[-1, 1].  The seed gives the order of the row lengths, the
columns, the values and the dense operands; sizes are the case's.
"""
from __future__ import annotations

import math

import torch

from segscan_gb300 import api, autograd, autotune
from segscan_gb300.batched import BatchedSpMM

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
SIZE = {"f32": 4, "bf16": 2, "f16": 2}

# the reference README's best static tuples at N = 64, as a program that calls the
# reference-named launchers has them in its source
LAUNCHERS = {
    "ebpr": (api.csrspmm_parreduce_nnzbalance_cg,
             dict(group_factor=5, thread_per_block=256, tile_factor=5, block_numer=1, block_denom=8)),
    "rbpr": (api.csrspmm_parreduce_rowbalance_cg,
             dict(group_factor=3, thread_per_block=256, tile_factor=3, block_numer=1, block_denom=2)),
    "ebsr": (api.csrspmm_rowcaching_nnzbalance_cg,
             dict(group_factor=4, thread_per_block=256, CoarsenFactor=4, ThreadNz=2, block_numer=1,
                  block_denom=16)),
    "rbsr": (api.csrspmm_seqreduce_rowbalance_cg,
             dict(coarsen_factor=4, thread_per_block=256, tile_factor=5, block_numer=1, block_denom=1)),
}


def listed():
    return [
        # a small graph's layer in a launch-bound loop (serving): one bound
        # plan, one C call per pass; the Poisson 4096 configuration
        dict(name="plan_poisson_4096_n16", kind="plan", law="poisson", rows=4096, cols=4096, mean=16.0, N=16,
             dtype="f32", out="f32"),
        # the headline workload through the default call: a million-row graph
        # with Zipf 2.1 row lengths, 64 features
        dict(name="spmm_powerlaw_1e6_n64", kind="spmm", law="powerlaw", rows=1_000_000, cols=1_000_000, alpha=2.1,
             lmax=20_000, N=64, dtype="f32", out="f32"),
        # the same graph with 16-bit storage and 128 features, the layout the
        # heuristic picks for that type
        dict(name="plan_powerlaw_1e6_n128_bf16", kind="plan", law="powerlaw", rows=1_000_000, cols=1_000_000,
             alpha=2.1, lmax=20_000, N=128, dtype="bf16", out="f32"),
        # few columns (class scores, label propagation) on the same graph
        dict(name="plan_powerlaw_1e6_n4", kind="plan", law="powerlaw", rows=1_000_000, cols=1_000_000, alpha=2.1,
             lmax=20_000, N=4, dtype="f32", out="f32"),
        # a regular banded matrix (finite elements), where the heuristic takes
        # the row-balanced strategy
        dict(name="plan_banded_120k_n64", kind="plan", law="banded", rows=120_000, cols=120_000, per_row=20,
             halfwidth=500, N=64, dtype="f32", out="f32"),
        # a program ported from the reference: its launcher name and tuple,
        # C zeroed by the caller, rectangular matrix and an odd width
        dict(name="launcher_ebsr_333k_n47", kind="launcher", strategy="ebsr", law="powerlaw", rows=333_337,
             cols=250_007, alpha=1.9, lmax=3_000, N=47, dtype="f32", out="f32"),
        # message aggregation of a GNN layer: sorted segment sum over the
        # million-row graph's edges
        dict(name="segment_sum_1e6_n64", kind="segment", reduce="sum", law="powerlaw", rows=1_000_000,
             cols=1_000_000, alpha=2.1, lmax=20_000, N=64, dtype="f32", out="f32"),
        # mean pooling of 16-bit features, ragged sizes
        dict(name="segment_mean_60k_n100_bf16", kind="segment", reduce="mean", law="poisson", rows=60_013,
             cols=60_013, mean=12.0, N=100, dtype="bf16", out="f32"),
        # training step with learned edge weights: forward and both gradients,
        # the largest configuration (2e6 rows, 128 features)
        dict(name="train_both_2e6_n128", kind="train", wants="both", law="powerlaw", rows=2_000_000,
             cols=2_000_000, alpha=2.1, lmax=50_000, N=128, dtype="f32", out="f32"),
        # training step of a graph convolution: fixed edge weights, gradient of
        # the 16-bit features only
        dict(name="train_B_300k_n64_bf16", kind="train", wants="B", law="powerlaw", rows=300_000, cols=300_000,
             alpha=1.8, lmax=5_000, N=64, dtype="bf16", out="f32"),
        # loading a graph: edge list in any order to CSR, then its transpose
        dict(name="load_powerlaw_1e6", kind="load", law="powerlaw", rows=1_000_000, cols=1_000_000, alpha=2.1,
             lmax=20_000, N=1, dtype="f32", out="f32"),
        # many small graphs per step: one batched launch replayed from a graph
        dict(name="batched_64_n64", kind="batched", count=64, rows_lo=100, rows_hi=50_000, alpha=2.3, lmax=2_000,
             N=64, dtype="f32", out="f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan", "plan", "spmm", "spmm", "launcher", "segment", "segment", "train", "train", "load",
                       "batched"])
    dtype = rng.choice(["f32", "f32", "bf16", "f16"])
    # widths a program has: powers of two, other multiples of four, odd ones
    N = rng.choice([2 ** rng.randint(0, 7), 4 * rng.randint(1, 32), rng.randint(1, 128)])
    c = dict(kind=kind, N=N, dtype=dtype, out="f32")
    if kind == "batched":
        hi = _log(rng, 2_000, 50_000)
        c.update(count=rng.randint(4, 64), rows_lo=100, rows_hi=hi, alpha=rng.choice([2.1, 2.3, 2.6]), lmax=2_000)
        return c
    rows = _log(rng, 1_000, 2_000_000)
    cols = max(64, min(2_000_000, int(rows * rng.choice([1.0, 1.0, 0.5, 1.7]))))
    law = rng.choice(["powerlaw", "powerlaw", "poisson", "banded"])
    c.update(law=law, rows=rows, cols=rows if law == "banded" else cols)
    if law == "powerlaw":
        alpha = rng.choice([1.9, 2.1, 2.3, 2.6])
        c.update(alpha=alpha, lmax=max(8, min(20_000, rows // 20) if alpha > 2 else min(2_000, rows // 20)))
    elif law == "poisson":
        c.update(mean=rng.choice([1.5, 4.0, 12.0, 16.0]))
    else:
        c.update(per_row=rng.choice([5, 10, 20]), halfwidth=rng.choice([50, 500]))
    # no more nonzeros than the largest listed matrix has
    c["rows"] = max(1_000, min(rows, int(9_000_000 / _mean(c))))
    c["cols"] = c["rows"] if law == "banded" else cols
    if kind == "launcher":
        # the row-balanced launchers walk a long row alone: used on regular rows
        c["strategy"] = rng.choice(["ebpr", "ebsr"] if law == "powerlaw" else ["ebpr", "ebsr", "rbpr", "rbsr"])
        c["N"] = max(2, N)
    elif kind == "spmm":
        # the result in the storage type, or FP32
        c["out"] = rng.choice([dtype, "f32"])
    elif kind == "segment":
        c["reduce"] = rng.choice(["sum", "sum", "mean", "max"])
    elif kind == "train":
        c["wants"] = rng.choice(["both", "B", "values"])
    elif kind == "load":
        c["dtype"] = "f32"
        c["N"] = 1
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(shape, g, dtype=torch.float32):
    return (torch.rand(shape, generator=g, device="cuda") * 2.0 - 1.0).to(dtype)


def _cdf(c):
    """P(length <= k) of a row's length, k from 0; what is above the last k is clipped to it."""
    if c["law"] == "powerlaw":
        k = torch.arange(1, c["lmax"] + 1, dtype=torch.float64)
        w = k.pow(-c["alpha"])
        tail = (c["lmax"] + 0.5) ** (1.0 - c["alpha"]) / (c["alpha"] - 1.0)
        cdf = torch.cumsum(w, 0) / (w.sum() + tail)
        return torch.cat([torch.zeros(1, dtype=torch.float64), cdf])
    if c["law"] == "poisson":
        k = torch.arange(0, int(c["mean"] * 4) + 16, dtype=torch.float64)
        return torch.cumsum(torch.exp(k * math.log(c["mean"]) - c["mean"] - torch.lgamma(k + 1)), 0)
    return torch.arange(0, c["per_row"] + 1, dtype=torch.float64) >= c["per_row"]


def _mean(c):
    """Expected row length."""
    return float((1.0 - _cdf(c)[:-1].double()).sum())


def _lengths(c):
    """Row lengths at evenly spaced quantiles of their law, so that a case has one number of
    nonzeros; in ascending order."""
    cdf = _cdf(c).double().cuda()
    u = (torch.arange(c["rows"], dtype=torch.float64, device="cuda") + 0.5) / c["rows"]
    return torch.searchsorted(cdf, u).clamp_(max=min(len(cdf) - 1, c["cols"]))


def _csr(c, g, dtype):
    """The case's matrix and the row of each nonzero.  Rows take the lengths in random order; a
    row of length L draws one column from each L-th part of its range (all columns, or the
    band), so columns are sorted and distinct."""
    M, K = c["rows"], c["cols"]
    lengths = _lengths(c)[torch.randperm(M, generator=g, device="cuda")]
    indptr = torch.zeros(M + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lengths, 0, out=indptr[1:])
    rows = torch.repeat_interleave(torch.arange(M, device="cuda"), lengths)
    j, L = torch.arange(rows.numel(), device="cuda") - indptr[rows], lengths[rows]
    width = min(2 * c["halfwidth"] + 1, K) if c["law"] == "banded" else K
    lo, hi = j * width // L, (j + 1) * width // L
    cols = lo + (torch.rand(rows.shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo)).long()
    if c["law"] == "banded":
        cols += (rows - c["halfwidth"]).clamp_(0, K - width)
    values = _uniform(rows.shape, g, dtype)
    return api.CsrMatrix(M, K, indptr.int(), cols.int(), values), rows


def _sizes(c):
    """Row counts of a batch, evenly spread over the logarithm of their range."""
    lo, hi, n = math.log(c["rows_lo"]), math.log(c["rows_hi"]), c["count"]
    return [int(math.exp(lo + (i + 0.5) / n * (hi - lo))) for i in range(n)]


def _batch(c, seed):
    dtype, g = DTYPES[c["dtype"]], _gen(seed)
    mats, Bs = [], []
    for m in _sizes(c):
        A, _ = _csr(dict(law="powerlaw", rows=m, cols=m, alpha=c["alpha"], lmax=min(c["lmax"], m)), g, dtype)
        mats.append(A)
        Bs.append(_uniform((m, c["N"]), g, dtype))
    return mats, Bs


def _inputs(c, seed):
    """The operands of every kind but the batch, as a dict."""
    dtype, g, N = DTYPES[c["dtype"]], _gen(seed), c["N"]
    A, rows = _csr(c, g, dtype)
    s = {"A": A}
    if c["kind"] == "segment":
        s["index"] = rows.int()
        s["src"] = _uniform((A.nnz, N), g, dtype)
    elif c["kind"] == "load":
        order = torch.randperm(A.nnz, generator=g, device="cuda")
        s["rows"] = rows.int()[order].contiguous()
        s["cols"] = A.indices[order].contiguous()
        s["values"] = A.values[order].contiguous()
    else:
        s["B"] = _uniform((c["cols"], N), g, dtype)
        if c["kind"] == "train":
            s["dC"] = _uniform((c["rows"], N), g)
    return s


def prepare(case, seed):
    c = dict(case)
    kind, N = c["kind"], c["N"]
    if kind == "batched":
        mats, Bs = _batch(c, seed)
        strategies, knobs = autotune.batch_plan(mats, N)
        plan = BatchedSpMM(mats, Bs, DTYPES[c["out"]], knobs, strategies=strategies)
        plan.capture()
        return {"case": c, "plan": plan}
    s = _inputs(c, seed)
    s["case"] = c
    A = s["A"]
    if kind == "plan":
        strategy, kw = autotune.heuristic(autotune.features(A), N, A.dtype)
        s["plan"] = api.SpmmPlan(A, N, strategy, api.make_knobs(strategy, N, **kw), DTYPES[c["out"]])
        s["out"] = torch.zeros((A.nrow, N), dtype=DTYPES[c["out"]], device="cuda")
    elif kind == "launcher":
        s["out"] = torch.zeros((A.nrow, N), device="cuda")
    elif kind == "train":
        # a training program builds the pattern and its transpose once
        s["pattern"] = autograd.pattern(A)
        s["pattern"].transposed()
        s["values"] = A.values.requires_grad_(c["wants"] != "B")
        s["B"].requires_grad_(c["wants"] != "values")
    return s


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "plan":
        return state["plan"].run(state["B"], state["out"])
    if kind == "spmm":
        return api.spmm(state["A"], state["B"], out_dtype=DTYPES[c["out"]])
    if kind == "launcher":
        call, knobs = LAUNCHERS[c["strategy"]]
        state["out"].zero_()
        call(state["A"], c["N"], state["B"], state["out"], **knobs)
        return state["out"]
    if kind == "segment":
        return api.segment(state["src"], state["index"], c["rows"], c["reduce"])
    if kind == "train":
        leaves = [t for t in (state["values"], state["B"]) if t.requires_grad]
        C = autograd.spmm(state["A"], state["values"], state["B"], pattern=state["pattern"])
        return [C.detach(), *torch.autograd.grad(C, leaves, state["dC"])]
    if kind == "load":
        A, perm = api.coo_to_csr(c["rows"], state["rows"], state["cols"], c["cols"], state["values"])
        AT, t_perm = api.transpose(A)
        return [A.indptr, A.indices, A.values, perm, AT.indptr, AT.indices, AT.values, t_perm]
    return state["plan"].replay()


# ---------------------------------------------------------------------------
# what a pass cannot do without, and what it gives in 64 bits
# ---------------------------------------------------------------------------
def _spmm_work(M, K, nnz, N, s, out):
    used = K * -math.expm1(-nnz / K)  # distinct columns of uniform draws
    return nnz * (4 + s) + 4 * (M + 1) + used * N * s + M * N * out, 2 * nnz * N


def work(case):
    c = case
    N, s, out = c["N"], SIZE[c["dtype"]], SIZE[c["out"]]
    if c["kind"] == "batched":
        mean = _mean(dict(law="powerlaw", alpha=c["alpha"], lmax=c["lmax"]))
        b, f = zip(*(_spmm_work(m, m, m * mean, N, s, out) for m in _sizes(c)))
        return {"bytes": sum(b), "flops": sum(f)}
    M, K = c["rows"], c["cols"]
    nnz = int(M * _mean(c))
    if c["kind"] == "segment":
        return {"bytes": nnz * (4 + N * s) + M * N * out, "flops": nnz * N}
    if c["kind"] == "load":
        # edges in; CSR with its permutation out, the transpose with its own out
        return {"bytes": nnz * (8 + s) + 2 * nnz * (8 + s) + 4 * (M + K + 2), "flops": 0}
    b, f = _spmm_work(M, K, nnz, N, s, out)
    if c["kind"] == "train":
        b += M * N * 4  # dC
        if c["wants"] != "values":  # the transposed pattern with its permutation, and dB
            b += 8 * nnz + 4 * (K + 1) + K * N * s
            f += 2 * nnz * N
        if c["wants"] != "B":  # the values' gradient
            b += nnz * s
            f += 2 * nnz * N
    return {"bytes": b, "flops": f}


def _product(A, B, transpose=False):
    v = A.values.detach().double()
    rows = torch.repeat_interleave(torch.arange(A.nrow, device="cuda"), torch.diff(A.indptr).long())
    i, j = (A.indices.long(), rows) if transpose else (rows, A.indices.long())
    out = torch.zeros((A.ncol if transpose else A.nrow, B.shape[1]), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 27) // max(1, B.shape[1]))
    for p in range(0, A.nnz, step):
        q = slice(p, p + step)
        out.index_add_(0, i[q], v[q, None] * B.detach()[j[q]].double())
    return out


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "batched":
        return [_product(A, B) for A, B in zip(*_batch(c, seed))]
    s = _inputs(c, seed)
    A = s["A"]
    if c["kind"] == "load":
        order = torch.argsort(s["rows"].long(), stable=True)
        values = s["values"][order].double()
        t_order = torch.argsort(s["cols"][order].long(), stable=True)
        return [None, None, values, None, None, None, values[t_order], None]
    if c["kind"] == "segment":
        src, index = s["src"], s["index"].long()
        out = torch.full((c["rows"], c["N"]), 0.0, dtype=torch.float64, device="cuda")
        step = max(1, (1 << 27) // c["N"])
        if c["reduce"] == "max":
            out.index_reduce_(0, index, src.double(), "amax", include_self=False)
            return out
        for p in range(0, A.nnz, step):
            out.index_add_(0, index[p:p + step], src[p:p + step].double())
        if c["reduce"] == "mean":
            out /= torch.bincount(index, minlength=c["rows"]).clamp(min=1)[:, None]
        return out
    C = _product(A, s["B"])
    if c["kind"] != "train":
        return C
    got = [C]
    if c["wants"] != "B":
        rows = torch.repeat_interleave(torch.arange(A.nrow, device="cuda"), torch.diff(A.indptr).long())
        dv = torch.empty(A.nnz, dtype=torch.float64, device="cuda")
        step = max(1, (1 << 27) // c["N"])
        for p in range(0, A.nnz, step):
            q = slice(p, p + step)
            dv[q] = (s["dC"][rows[q]].double() * s["B"][A.indices[q].long()].double()).sum(1)
        got.append(dv)
    if c["wants"] != "values":
        got.append(_product(A, s["dC"], transpose=True))
    return got
