"""What a tensor-core build leaves allocated: nothing of its candidate queue.

The queue (64 million pairs, 805 MB) is needed while joining only; a context
that has built with the filter holds what one that has built in FP32 holds, but
for the small counters and the audit's statistics.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["bf16", "fp8_always"])
def test_candidate_queue_is_given_back(mode):
    import torch

    from kgraph_b200 import capi
    X = np.random.default_rng(0).standard_normal((20_000, 64)).astype(np.float32)
    kept = {}
    for m in ("fp32", mode):
        ctx = capi.Context(0)
        try:
            ctx.set_data(X, "euclidean")
            ctx.set_join_precision(m)
            ctx.build(iterations=2, K=10, L=20, S=5)   # the kernels' own memory, for both
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            for _ in range(2):
                ctx.build(iterations=6, K=25, L=50, S=10)
            torch.cuda.synchronize()
            kept[m] = before - torch.cuda.mem_get_info()[0]
            if m == mode:
                assert ctx.join_stats()["tc_iterations"] > 0
        finally:
            ctx.close()
        first = capi.Context(0)
        try:
            first.set_data(X, "euclidean")
            first.set_join_precision(m)
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            first.build(iterations=6, K=25, L=50, S=10)
            torch.cuda.synchronize()
            kept[m + " first"] = before - torch.cuda.mem_get_info()[0]
        finally:
            first.close()
    assert kept[mode] - kept["fp32"] < 100 << 20, kept
    assert kept[mode + " first"] - kept["fp32 first"] < 100 << 20, kept
