"""Which rows and lists the tensor-core join takes: two 128-row tiles, a row and
28 bytes per list entry within 200 KB, to the entry; the rest is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# lists of max(2 S, L) + R new and L + R old entries: 40 + 2 R at L = 20, S = 5
@pytest.mark.parametrize("mode,d,R,taken", [
    ("fp8_always", 20, 3488, True),      # 8,192 + 128 + 28 x 7,016 bytes
    ("fp8_always", 20, 3489, False),
    ("bf16_always", 380, 98, True),      # 196,608 + 1,536 + 28 x 236
    ("bf16_always", 380, 99, False),
    ("bf16_always", 16, 3489, True),     # 8,192 + 64 + 28 x 7,018
    ("bf16_always", 16, 3490, False),
])
def test_longest_lists(mode, d, R, taken):
    from kgraph_b200 import capi
    rng = np.random.default_rng(d)
    n = 1200
    X = rng.standard_normal((n, d)).astype(np.float32)
    ctx = capi.Context(0)
    try:
        ctx.set_data(X, "l2sqr")
        ctx.set_join_precision(mode)
        kw = dict(iterations=2, K=10, L=20, S=5, R=R, delta=0.0, recall=2.0, controls=10)
        if not taken:
            with pytest.raises(capi.KGError, match="fit in shared memory"):
                ctx.build(**kw)
            return
        ctx.build(**kw)
        st = ctx.join_stats()
        assert st["tc_iterations"] == 2 and st["violations"] == 0
        off, ids, dists, _ = ctx.graph()
        for r in (0, n // 2, n - 1):
            a, b = int(off[r]), int(off[r + 1])
            dd = ((X[ids[a:b]].astype(np.float64) - X[r]) ** 2).sum(1)
            assert b - a >= 10 and np.allclose(dd, dists[a:b], rtol=1e-5)
    finally:
        ctx.close()
