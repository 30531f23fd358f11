"""The warp's introsort (kg_sort.h warp_gnu_sort), through the two callers.

Reverse completion sorts each node's list with it: lists of every length around
its piece (32), its ranges (16), the shared-memory capacity (480) and its limit
(8,191), with few distinct distances, sorted and organ-pipe orders, self loops
and repeated edges, must come out as the reference's std::sort and std::unique
leave them -- the oracle's serial restatement, bit for bit.  The search sorts its
seed pool with it: many tied seeds must give the oracle's walk.
"""
import numpy as np
import pytest

from oracle import kgoracle as ko

pytestmark = pytest.mark.gpu


def hub_graph(rng, sizes, values):
    """Node h < len(sizes) is pointed at by `sizes[h]` other nodes; distances from few values."""
    hubs = len(sizes)
    n = max(sizes) + hubs + 40
    rows = [[] for _ in range(n)]
    for h, s in enumerate(sizes):
        for src in rng.choice(np.arange(hubs, n), s, replace=False):
            rows[src].append(h)
    for h in range(hubs):   # the hubs' own edges, self loops and repeats among them
        rows[h] = [h, h] + list(rng.integers(0, n, 20)) + [int(rng.integers(0, n))] * 2
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum([len(r) for r in rows])
    ids = np.concatenate([np.asarray(r, np.uint32) for r in rows])
    shape = rng.integers(0, 4)
    d = rng.integers(0, values, len(ids)).astype(np.float32)
    if shape == 1:
        d = np.sort(d)
    elif shape == 2:
        d = np.sort(d)[::-1].copy()
    elif shape == 3:
        d = np.concatenate([np.sort(d[::2]), np.sort(d[1::2])[::-1]])
    return ko.Graph(off, ids, d, np.diff(off).astype(np.uint32))


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("values", [2, 7, 100, 1 << 20])
def test_reverse_lists_of_every_length(gpu_ctx, seed, values):
    rng = np.random.default_rng(100 * seed + values)
    sizes = list(range(0, 70, 3)) + [94, 95, 96, 97, 126, 255, 300, 452, 453, 454, 455, 456, 457, 900, 2100]
    if seed == 0:
        sizes += [8164, 8165, 8166, 8167, 8168, 9000]
    G = hub_graph(rng, sizes, values)
    X = rng.random((len(G.M), 4), dtype=np.float32)
    gpu_ctx.set_data(X, "l2sqr")
    gpu_ctx.set_graph(G.offsets, G.ids, G.dists, G.M)
    gpu_ctx.reverse(-1)
    off, ids, d, M = gpu_ctx.graph()
    R = ko.Oracle(X, "l2sqr").reverse(G, -1)
    assert (off == R.offsets).all() and (M == R.M).all()
    assert (ids == R.ids).all()
    assert (d.view(np.uint32) == np.asarray(R.dists, np.float32).view(np.uint32)).all()


@pytest.mark.parametrize("P", [3, 16, 17, 33, 100, 1000, 2500])
def test_seed_pools_with_ties(gpu_ctx, P):
    rng = np.random.default_rng(P)
    n = 4000
    X = rng.integers(0, 3, (n, 5)).astype(np.float32)   # 243 distinct rows
    Q = rng.integers(0, 3, (12, 5)).astype(np.float32)
    deg = rng.integers(2, 30, n)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(deg)
    ids = rng.integers(0, n, int(off[-1])).astype(np.uint32)
    G = ko.Graph(off, ids, np.zeros(len(ids), np.float32), deg.astype(np.uint32))
    gpu_ctx.set_data(X, "l2sqr")
    gpu_ctx.set_graph(G.offsets, G.ids, G.dists, G.M)
    o = ko.Oracle(X, "l2sqr")
    oi, od, oc, ok = o.search(G, Q, K=5, P=P)
    try:
        for compact in (0, 1):
            gpu_ctx.set_search_tuning(4, 0, 2, 64, compact)
            gi, gd, gc, gk = gpu_ctx.search(Q, K=5, P=P)
            assert (gc == oc).all() and (gk == ok).all() and (gi == oi).all()
    finally:
        gpu_ctx.set_search_tuning(4, 0, 2)
