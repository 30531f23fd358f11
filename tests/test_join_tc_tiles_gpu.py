"""The tensor-core join's tiles (kg_join_tc.cu) against the warp join.

The first iteration evaluates every pair of every node's lists.  With 32 new
columns and 96 further partners a tile, list lengths around one, two and more
blocks of columns and one and two tiles of partners are covered, with FP32
pairs counted once each and every node's list ending with the same distances.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,d", [("bf16_always", 64), ("bf16_always", 100), ("fp8_always", 96)])
@pytest.mark.parametrize("metric", ["euclidean", "angular", "l2sqr"])
@pytest.mark.parametrize("S", [1, 15, 16, 17, 33, 64, 65])
def test_first_join_equals_warp_join(mode, d, metric, S):
    from kgraph_b200 import capi
    rng = np.random.default_rng(d * 100 + S)
    n = 500
    X = rng.standard_normal((n, d)).astype(np.float32)
    X[5] = X[6]
    out = {}
    for m in ("fp32", mode):
        ctx = capi.Context(0)
        try:
            capi.set_verbosity(0)
            ctx.set_data(X, metric)
            ctx.set_join_precision(m)
            ctx.set_join_inserts("locked")
            info = ctx.build(iterations=1, K=min(10, S), L=max(S, 40), S=S, R=10, delta=0.0, recall=2.0, controls=10)
            off, ids, dists, _ = ctx.graph()
            out[m] = (off, dists.view(np.uint32), ctx.build_work()[0], info["recall"], ctx.join_stats())
        finally:
            ctx.close()
    a, b = out["fp32"], out[mode]
    assert b[4]["tc_iterations"] == 1 and b[4]["violations"] == 0
    assert a[2] == b[2] > 0                 # pairs evaluated
    assert (a[0] == b[0]).all()             # list lengths
    assert (a[1] == b[1]).all()             # distances, bit for bit
    assert a[3] == b[3]
