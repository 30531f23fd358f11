"""Queries whose candidates from the sampled threshold outgrow their room.

Float rows in clusters a few spreads apart have a BF16 margin that is wide
beside the distances between neighbours: the sample (1/16 of the rows at
K = 10) leaves 16 K rows per query times what the margin adds, more than the
room of 1,024.  With all rows as the sample the margin's own rows fit, so no
query may be scanned in full; the results are the scan's.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mixture(torch, n, d, ratio, seed):
    g = torch.Generator(device="cuda").manual_seed(99)
    centres = torch.randn(64, d, device="cuda", generator=g) * ratio
    g.manual_seed(seed)
    lab = torch.randint(0, 64, (n,), device="cuda", generator=g)
    return (torch.randn(n, d, device="cuda", generator=g) + centres[lab]).contiguous()


# (full scans at 200k rows and 1,000 queries without the second pass: 605, 3, 106, 1)
@pytest.mark.parametrize("d,ratio,K,nq,host", [
    (128, 2.0, 10, 1000, False),
    (128, 2.0, 10, 20_000, False),   # more than one batch of queries that come again
    (128, 1.0, 100, 1000, True),
    (250, 1.5, 10, 1000, False),
    (128, 0.0, 10, 1000, True),
])
def test_overflowing_queries_take_all_rows_as_the_sample(d, ratio, K, nq, host):
    import ctypes as C

    import torch

    from kgraph_b200 import capi
    n = 200_000
    X, Q = mixture(torch, n, d, ratio, 1), mixture(torch, nq, d, ratio, 2)
    ctx = capi.Context(0)
    try:
        ctx.set_data(X, "euclidean")
        p = capi.SearchParams(K, 0, n, 10, 1, 1e30, 1998, 0)
        res = []
        for mode in ("tensor", "scan"):
            ctx.set_bruteforce_mode(mode)
            if host:
                res.append(ctx.search(Q.cpu().numpy(), K=K))
            else:
                o = [torch.zeros(nq, K, dtype=torch.int32, device="cuda"), torch.zeros(nq, K, device="cuda"),
                     torch.zeros(nq, dtype=torch.int32, device="cuda"), torch.zeros(nq, device="cuda")]
                ctx.search_raw(C.c_void_p(Q.data_ptr()), nq, Q.stride(0) * 4, p, None, None, K,
                               *[C.c_void_p(t.data_ptr()) for t in o])
                res.append([t.cpu().numpy() for t in o])
            if mode == "tensor":
                st = ctx.bruteforce_stats()
        assert st["tensor"] == 1 and st["full_scans"] == 0
        for a, b in zip(*res):
            assert np.array_equal(a, b)
    finally:
        ctx.close()


@pytest.mark.parametrize("metric", ["euclidean", "angular", "l2sqr"])
def test_the_margin_alone_outgrows_the_room(metric):
    """Half the rows and half the queries' neighbourhoods are one point: those queries are scanned in
    full after the second pass, the others are not."""
    from kgraph_b200 import capi
    rng = np.random.default_rng(3)
    X = rng.standard_normal((12_000, 24)).astype(np.float32)
    X[::2] = X[0]
    Q = rng.standard_normal((300, 24)).astype(np.float32)
    Q[::3] = X[0]
    ctx = capi.Context(0)
    try:
        ctx.set_data(X, metric)
        res = []
        for mode in ("scan", "tensor"):
            ctx.set_bruteforce_mode(mode)
            res.append(ctx.search(Q, K=5))
        st = ctx.bruteforce_stats()
        assert st["tensor"] == 1 and 100 <= st["full_scans"] < 300
        for a, b in zip(*res):
            assert np.array_equal(a, b)
    finally:
        ctx.close()
