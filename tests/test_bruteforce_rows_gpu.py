"""Device memory of the tensor-core brute force's copy of the dataset: its BF16
rows and, unless angular, 16 bytes per row for the norm's three parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["euclidean", "angular"])
def test_copy_of_the_rows(metric):
    import torch

    from kgraph_b200 import capi
    n, d = 2_000_000, 16
    X = torch.rand(n, d, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)) + 0.5
    Q = X[:3].cpu().numpy()
    warm, ctx = capi.Context(0), capi.Context(0)
    try:
        warm.set_data(X[:2000].contiguous(), metric)   # the kernels' own memory
        warm.set_bruteforce_mode("tensor")
        warm.search(Q, K=10)
        ctx.set_data(X, metric)
        ctx.set_bruteforce_mode("scan")
        a = ctx.search(Q, K=10)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        ctx.set_bruteforce_mode("tensor")
        b = ctx.search(Q, K=10)
        torch.cuda.synchronize()
        grown = before - torch.cuda.mem_get_info()[0]
        assert ctx.bruteforce_stats()["tensor"] == 1
        # three queries' work space is below 8 MB, allocations go in 2 MB pieces
        assert grown <= n * (2 * d + (0 if metric == "angular" else 16)) + (16 << 20), grown
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
    finally:
        ctx.close()
        warm.close()
