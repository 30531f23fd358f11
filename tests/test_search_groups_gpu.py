"""The walk's groups of candidates: batches of S neighbours read several at a time.

An entry's adjacency comes in windows of 128 ids, whose unvisited neighbours
are taken up to 32 at a time across batch borders and put back behind the batch
in which an insert lands at or before the expanded entry.  Batch sizes around
the group and window sizes, degrees above a window and above its list of 64
unvisited neighbours, and ids that recur within and between groups must give
the oracle's ids, distances, counts and cost.
"""
import numpy as np
import pytest

from oracle import kgoracle as ko

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("S", [1, 7, 31, 32, 33, 63, 65, 129, 200, 70000])
@pytest.mark.parametrize("spread", [60, 5000])   # ids from a range this wide around the node: many recur / few
def test_batches_groups_and_windows_match_oracle(gpu_ctx, S, spread):
    rng = np.random.default_rng(S + spread)
    n, d = 5000, 20
    X = rng.integers(0, 12, (n, d)).astype(np.float32)
    Q = rng.integers(0, 12, (24, d)).astype(np.float32)
    deg = rng.integers(1, 301, n)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(deg)
    src = np.repeat(np.arange(n), deg)
    ids = ((src + rng.integers(0, spread, len(src))) % n).astype(np.uint32)
    G = ko.Graph(off, ids, np.zeros(len(ids), np.float32), rng.integers(1, 301, n).astype(np.uint32))
    gpu_ctx.set_data(X, "euclidean")
    gpu_ctx.set_graph(G.offsets, G.ids, G.dists, G.M)
    o = ko.Oracle(X, "euclidean")
    try:
        for compact, kw in ((1, dict(K=10, P=40)), (0, dict(K=10, P=40)), (1, dict(K=3, P=400, M=300))):
            gpu_ctx.set_search_tuning(4, 0, 2, 64, compact)
            gi, gd, gc, gk = gpu_ctx.search(Q, S=S, **kw)
            oi, od, oc, ok = o.search(G, Q, S=S, **kw)
            assert (gc == oc).all() and (gk == ok).all()
            for q in range(len(Q)):
                assert (gi[q, :gc[q]] == oi[q, :gc[q]]).all(), q
                assert (bits(gd[q, :gc[q]]) == bits(od[q, :gc[q]])).all(), q
        gpu_ctx.set_search_precision("bf16")   # the filtered walk takes the same groups
        fi, fd, fc, fk = gpu_ctx.search(Q, K=10, P=40, S=S)
        oi, od, oc, ok = o.search(G, Q, K=10, P=40, S=S)
        assert (fc == oc).all() and (fk == ok).all() and all((fi[q, :fc[q]] == oi[q, :fc[q]]).all() for q in range(len(Q)))
    finally:
        gpu_ctx.set_search_precision("fp32")
        gpu_ctx.set_search_tuning(4, 0, 2)
