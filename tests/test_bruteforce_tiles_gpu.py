"""The brute-force sweeps at the edges of their tiles, against the CUDA-core scan.

Tiles are 128 or 256 queries by 256 rows in boxes of 64 columns; the sample is
all rows or a share of them, its maxima over 1, 4 or 32 rows.  Sizes around each
of these, every number of column boxes, and data or queries without a usable
error margin (infinities, NaN) must give the scan's ids, distances and counts.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def both(ctx, Q, K):
    out = []
    for mode in ("scan", "tensor"):
        ctx.set_bruteforce_mode(mode)
        out.append(ctx.search(Q, K=K))
    st = ctx.bruteforce_stats()
    ctx.set_bruteforce_mode("auto")
    (i1, d1, c1, k1), (i2, d2, c2, k2) = out
    assert (c1 == c2).all() and (bits(k1) == bits(k2)).all()
    for q in range(len(c1)):
        assert (i1[q, :c1[q]] == i2[q, :c1[q]]).all(), q
        assert (bits(d1[q, :c1[q]]) == bits(d2[q, :c1[q]])).all(), q
    return st


@pytest.mark.parametrize("n,d,K,nq", [
    (1, 3, 1, 1), (5, 16, 10, 3), (255, 17, 5, 127), (256, 64, 128, 128), (257, 65, 1, 129), (100, 40, 128, 300),
    (4095, 128, 2, 256), (4111, 129, 3, 257), (16385, 192, 10, 40), (33000, 193, 25, 130), (20000, 256, 128, 385),
    (70001, 20, 70, 1), (131077, 48, 16, 513),
])
@pytest.mark.parametrize("metric", ["euclidean", "angular", "l2sqr"])
def test_tile_edges_equal_scan(n, d, K, nq, metric):
    from kgraph_b200 import capi
    rng = np.random.default_rng(n + d + K + nq)
    # clustered: the rows of a cluster lie together, as in data written cluster by cluster
    X = (rng.integers(-30, 30, (max(1, n // 500), d))[np.arange(n) * max(1, n // 500) // n]
         + rng.integers(-6, 7, (n, d))).astype(np.float32)
    if n > 4:
        X[n // 2] = 0   # a zero row
    Q = X[rng.integers(0, n, nq)] + rng.integers(-3, 4, (nq, d)).astype(np.float32)
    if metric == "angular":
        X += rng.random((n, d), dtype=np.float32) * (X != 0)
    ctx = capi.Context(0)
    try:
        ctx.set_data(X, metric)
        assert both(ctx, Q, K)["tensor"] == 1
    finally:
        ctx.close()


@pytest.mark.parametrize("value", [np.inf, -np.inf, 3e38])
def test_data_and_queries_without_a_margin(value):
    """A row with an infinity, or values whose squares overflow, leaves no error
    bound: the batch is scanned.  A query with one is scanned, the others are not."""
    from kgraph_b200 import capi
    rng = np.random.default_rng(3)
    X = rng.random((3000, 24), dtype=np.float32)
    Q = rng.random((9, 24), dtype=np.float32)
    ctx = capi.Context(0)
    try:
        ctx.set_data(X, "l2sqr")
        Q2 = Q.copy()
        Q2[4, 7] = value
        st = both(ctx, Q2, 5)
        assert st["tensor"] == 1 and st["full_scans"] == 1
        X[77, 3] = value
        ctx.set_data(X, "l2sqr")
        assert both(ctx, Q, 5)["tensor"] == 0
    finally:
        ctx.close()
