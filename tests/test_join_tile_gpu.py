"""The register-tiled local join (kg_build.cu join_tile_kernel) against the warp join.

The first iteration's join is the same work in both insert modes: every node's
2 S random new entries, all pairs of them.  The warp join (locked inserts)
evaluates them one by one with pair_dist; the tiled join must evaluate the same
pairs to the same bits, so that every node's list ends with the same distances
whatever the order of the inserts.  List lengths around the tile's 4 x 32, rows
with tails, lists longer than the rows that fit in shared memory, and every
metric are covered.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["euclidean", "angular", "l2sqr"])
@pytest.mark.parametrize("d,S", [(7, 1), (16, 2), (24, 3), (31, 8), (40, 16), (128, 17), (130, 24), (100, 33), (320, 20),
                                 (600, 30), (1100, 6)])
def test_first_join_equals_warp_join(metric, d, S):
    from kgraph_b200 import capi
    rng = np.random.default_rng(d * 100 + S)
    n = 900 if d < 200 else 400
    X = rng.standard_normal((n, d)).astype(np.float32)
    X[5] = X[6]   # equal rows: distance ties, and zero under l2sqr
    out = {}
    for mode in ("locked", "deferred"):
        ctx = capi.Context(0)
        try:
            capi.set_verbosity(0)
            ctx.set_data(X, metric)
            ctx.set_join_inserts(mode)
            info = ctx.build(iterations=1, K=min(10, S), L=max(S, 40), S=S, R=10, delta=0.0, recall=2.0, controls=10)
            off, ids, dists, _ = ctx.graph()
            out[mode] = (off, dists.view(np.uint32), ctx.build_work()[0], info["recall"])
        finally:
            ctx.close()
    a, b = out["locked"], out["deferred"]
    assert a[2] == b[2] > 0                 # pairs evaluated
    assert (a[0] == b[0]).all()             # list lengths
    assert (a[1] == b[1]).all()             # distances, bit for bit
    assert a[3] == b[3]
