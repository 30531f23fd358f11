"""The tensor-core join's filter as it runs: builds of several filtered iterations.

From the second iteration on the radii are finite and most pairs are skipped;
the audit evaluates the filter's own bound and decision on every pair of the
sampled nodes (1 in 2,048) and must find no violation.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["bf16_always", "fp8_always"])
@pytest.mark.parametrize("metric", ["euclidean", "angular", "l2sqr"])
@pytest.mark.parametrize("kind,d", [("mixture", 64), ("mixture", 128), ("offset", 96)])
def test_no_pair_of_a_sampled_node_is_lost(mode, metric, kind, d):
    from kgraph_b200 import capi
    rng = np.random.default_rng(d)
    n = 30_000
    X = (rng.standard_normal((60, d))[rng.integers(0, 60, n)] * 2 + rng.standard_normal((n, d))).astype(np.float32)
    if kind == "offset":
        X += 20
    X[100:200] = X[300:400]   # equal rows
    ctx = capi.Context(0)
    try:
        ctx.set_data(X, metric)
        ctx.set_join_precision(mode)
        ctx.build(iterations=8, K=20, L=40, S=10, R=40, delta=0.0, recall=2.0)
        st = ctx.join_stats()
        assert st["tc_iterations"] == 8
        skipped = 1 - st["rechecked"] / st["pairs"]
        assert skipped > 0.02, st
        assert st["sampled"] > 3000 and st["violations"] == 0, st
    finally:
        ctx.close()
