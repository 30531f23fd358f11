"""The tensor-core brute force's work space does not grow with rows times queries.

A query's group maxima take up to n / 32 floats, so a large exact search is cut
into batches by bytes.  One call of 32,768 queries, K = 128, on 4 million rows
(4.1 GB of maxima at once) must stay within the batch's half gigabyte plus what
grows with one factor only, and the batches' results must be the scan's.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_search_runs_in_batches_of_bounded_memory():
    import ctypes as C

    import torch

    from kgraph_b200 import capi
    n, d, K, nq = 4_000_000, 16, 128, 32768
    g = torch.Generator(device="cuda").manual_seed(5)
    X = torch.rand(n, d, device="cuda", generator=g)
    Q = torch.rand(nq, d, device="cuda", generator=g)
    out = [torch.zeros(nq, K, dtype=torch.int32, device="cuda"), torch.zeros(nq, K, device="cuda"),
           torch.zeros(nq, dtype=torch.int32, device="cuda"), torch.zeros(nq, device="cuda")]
    ctx = capi.Context(0)
    try:
        ctx.set_data(X, "l2sqr")
        ctx.set_bruteforce_mode("tensor")
        p = capi.SearchParams(K, 0, n, 10, 1, 1e30, 1998, 0)

        def run(q, o):
            ptrs = [C.c_void_p(t.data_ptr()) for t in o]
            ctx.search_raw(C.c_void_p(q.data_ptr()), q.shape[0], q.stride(0) * 4, p, None, None, K, *ptrs)

        run(Q[:1], [t[:1] for t in out])   # the walk's and the dataset's own buffers
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        run(Q, out)
        torch.cuda.synchronize()
        grown = before - torch.cuda.mem_get_info()[0]
        assert ctx.bruteforce_stats()["tensor"] == 1
        # a batch's maxima and candidates 512 MB, twice that for what the segments' room adds
        assert grown < 1 << 30, grown
        ctx.set_bruteforce_mode("scan")
        at = torch.tensor([0, 1, 255, 9999, 13055, 13056, 13057, 20001, 26111, 26112, 32767], device="cuda")
        q = Q[at].contiguous()
        ref = [torch.zeros_like(t[at]) for t in out]
        run(q, ref)
        torch.cuda.synchronize()
        for a, b in zip(out, ref):
            assert torch.equal(a[at], b)
        assert np.array_equal(out[2].cpu().numpy(), np.full(nq, K))
    finally:
        ctx.close()
