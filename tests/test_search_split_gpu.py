"""The D-split a search takes when no shape was chosen (kg_search.cu search_split):
2 lanes per distance on narrow rows, 4 on wide ones; a chosen shape is kept, and
the results are the same bits either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,filt,nq,split", [(5, "fp32", 3, 2), (63, "fp32", 9, 2), (64, "fp32", 9, 4), (128, "fp32", 9, 4),
                                             (96, "bf16", 9, 2), (97, "bf16", 9, 4), (31, "fp8", 2000, 2),
                                             (32, "fp8", 2000, 4), (96, "fp8", 9, 2), (112, "fp8", 9, 4)])
def test_split_without_a_chosen_shape(d, filt, nq, split):
    from kgraph_b200 import capi
    rng = np.random.default_rng(d)
    n = 3000
    X = rng.integers(0, 9, (n, d)).astype(np.float32)
    Q = rng.integers(0, 9, (nq, d)).astype(np.float32)
    off = np.arange(0, 20 * n + 1, 20).astype(np.uint64)
    ids = rng.integers(0, n, 20 * n).astype(np.uint32)
    ctx = capi.Context(0)
    try:
        ctx.set_data(X, "euclidean")
        ctx.set_graph(off, ids, None, np.full(n, 20, np.uint32))
        ctx.set_search_precision(filt)
        assert ctx.search_tuning()["split"] == 4
        a = ctx.search(Q, K=10, P=30)
        assert ctx.last_search_shape()["split"] == split
        for chosen in (4, 2, 8):
            ctx.set_search_tuning(chosen, 0, 2, 64, 1)
            b = ctx.search(Q, K=10, P=30)
            assert ctx.last_search_shape()["split"] == chosen
            for x, y in zip(a, b):
                assert (np.asarray(x).view(np.uint32) == np.asarray(y).view(np.uint32)).all()
    finally:
        ctx.close()
