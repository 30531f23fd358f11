"""The narrow rows' local join (kg_build.cu join_lane_kernel) against the warp join.

As for the tiled join: the first iteration's join is the same work in both insert
modes, so every node's list must end with the same distances, to the bit.  Row
widths with and without a tail on both sides of 8, lists around the 16 and 32 new
entries and the 32 and 64 partners of a pass, several rounds of nodes, and every
metric are covered.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["euclidean", "angular", "l2sqr"])
@pytest.mark.parametrize("d", [1, 7, 8, 16, 17, 24, 32, 45, 48, 57, 64])
@pytest.mark.parametrize("S,cap", [(1, 0), (8, 0), (16, 0), (17, 40000), (33, 0), (70, 0)])
def test_first_join_equals_warp_join(metric, d, S, cap):
    from kgraph_b200 import capi
    rng = np.random.default_rng(d * 100 + S)
    n = 700 if S < 20 else 300
    X = rng.integers(-2, 3, (n, d)).astype(np.float32) if d < 9 else rng.standard_normal((n, d)).astype(np.float32)
    X[5] = X[6]
    X[7] = 0.0
    out = {}
    for mode in ("locked", "deferred"):
        ctx = capi.Context(0)
        try:
            capi.set_verbosity(0)
            ctx.set_data(X, metric)
            ctx.set_join_inserts(mode)
            if cap and mode == "deferred":
                ctx.set_join_offer_capacity(cap)
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
