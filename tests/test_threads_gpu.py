"""Host threads with matrices of different sizes in the kernels whose shared memory follows the size
(staged rbsr, COO -> CSR, transpose): no call is refused and every result is that of a call alone, bit for
bit."""
import threading

import numpy as np
import pytest
import torch

from gpu_util import dev_csr
from segscan_gb300 import synth

pytestmark = pytest.mark.gpu


def test_sizes_side_by_side(cuda):
    from segscan_gb300 import api
    rng = np.random.default_rng(3)
    jobs = []
    for M in (16_000, 60_000):  # N = 32: 81,600 and 104,448 bytes a block
        A = dev_csr(synth.poisson(M, M, 12.0, seed=M))
        B = torch.rand(M, 32, device="cuda")
        jobs.append(lambda s, A=A, B=B: [api.spmm(A, B, "rbsr", stream=s)])
        AT = A
        jobs.append(lambda s, A=AT: [*(lambda T, p: (T.indptr, T.indices, p))(*api.transpose(A, stream=s))])
    for nrow, nnz in ((3_000, 40_000), (400_000, 1_500_000)):
        rows = torch.from_numpy(rng.integers(0, nrow, nnz).astype(np.int32)).cuda()
        cols = torch.from_numpy(rng.integers(0, nrow, nnz).astype(np.int32)).cuda()
        jobs.append(lambda s, n=nrow, r=rows, c=cols: [
            *(lambda A, p: (A.indptr, A.indices, p))(*api.coo_to_csr(n, r, c, ncol=n, stream=s))])
    want = [[t.clone() for t in job(None)] for job in jobs]
    torch.cuda.synchronize()
    errors = []

    def work(job, ref):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for _ in range(40):
                    got = job(s)
                s.synchronize()
                assert all(torch.equal(a, b) for a, b in zip(got, ref))
        except Exception as exc:  # surfaced in the main thread
            errors.append(exc)

    threads = [threading.Thread(target=work, args=x) for x in zip(jobs, want)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors
