"""Device memory of reverse completion: 32 bytes per forward edge of work space
(target, source and distance, both again sorted, the assembled distances; the
assembled ids take the unsorted values' place), 48 per node, the sort's own, and
the completed graph, each with an eighth of slack at most."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_work_space_per_edge():
    import torch

    from kgraph_b200 import capi
    n, M = 100_000, 100
    rng = np.random.default_rng(0)
    ids = rng.integers(0, n, (n, M), dtype=np.uint32)
    ctx = capi.Context(0)
    try:
        ctx.set_data(rng.random((n, 4), dtype=np.float32), "l2sqr")
        small = rng.integers(0, n, (n, 1), dtype=np.uint32)   # the kernels' own memory
        ctx.set_graph(np.arange(n + 1), small, np.zeros((n, 1), np.float32), np.ones(n))
        ctx.reverse(-1)
        ctx.set_graph(np.arange(0, n * M + 1, M), ids, rng.random((n, M), dtype=np.float32), np.full(n, M))
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        ctx.reverse(-1)
        torch.cuda.synchronize()
        grown = before - torch.cuda.mem_get_info()[0]
        edges, final = n * M, len(ctx.graph()[1])
        # the sort's own space is a few counters per tile of keys (1 MB here), allocations go in 2 MB pieces
        bound = (32 * edges + 48 * n + 8 * final) * 9 // 8 + (64 << 20)
        assert grown <= bound, (grown, bound)
    finally:
        ctx.close()
