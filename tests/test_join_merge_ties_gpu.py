"""The deferred merge of pools with many offers of equal distance.

Up to 512 offers that no cut between distances separates still go in ascending
(distance, id) order, in passes of at most 256: one distance, copies of one
offer beyond a pass, and both among spread ones, against the oracle's serial
inserts in that order, bit for bit.
"""
import numpy as np
import pytest

from test_join_merge_gpu import FLAG, FMAX, UNSET_ID, UU, _serial

pytestmark = pytest.mark.gpu


def case(seed, n, L, m, ids, distances, copies):
    """n pools of 0 to L entries; m offers each, distances from `distances` (a fixed one per pair),
    a share `copies` of them repeats of a few ids."""
    rng = np.random.default_rng(seed)
    table = rng.choice(np.asarray(distances, np.float32), (n, ids))
    pool_d = np.full((n, L + 1), FMAX, np.float32)
    pool_i = np.full((n, L + 1), UNSET_ID, np.uint32)
    nodeL = np.zeros(n, np.uint32)
    radius = np.full(n, FMAX, np.float32)
    tg, cd = [], []
    for x in range(n):
        Lc = [0, L // 2, L, L][x % 4]
        members = rng.choice([c for c in range(ids) if c != x], Lc, replace=False)
        members = members[np.argsort(table[x, members], kind="stable")]
        pool_d[x, :Lc] = table[x, members]
        pool_i[x, :Lc] = members.astype(np.uint32) | np.uint32(FLAG)
        nodeL[x] = Lc
        if x % 4 == 3:
            radius[x] = pool_d[x, L - 1]
        pick = rng.integers(0, ids, m)
        few = rng.integers(0, ids, 2)
        pick = np.where(rng.random(m) < copies, rng.choice(few, m), pick)
        pick = pick[pick != x]
        tg += [x] * len(pick)
        cd += list(pick)
    tg, cd = np.array(tg, np.uint32), np.array(cd, np.uint32)
    h = (tg.astype(np.uint64) * 7919 + cd.astype(np.uint64) * 104729) & 0xFFFFFFFF
    sr = (h % n).astype(np.uint32) | np.where((h >> 7) & 1, UU, 0).astype(np.uint32)
    return pool_d, pool_i, nodeL, radius, tg, cd, table[tg, cd], sr


@pytest.mark.parametrize("seed,L,K,m,ids,distances,copies", [
    (1, 100, 50, 400, 5000, [3], 0.0),            # one distance, two passes' worth
    (2, 100, 50, 512, 5000, [3, 4], 0.0),
    (3, 100, 50, 512, 5000, [3], 0.0),            # as many as go in order
    (4, 40, 20, 257, 600, [0], 0.0),
    (5, 40, 20, 500, 600, [6], 0.6),              # hundreds of copies of two offers
    (6, 16, 8, 512, 900, [7], 1.0),               # nothing but copies
    (7, 100, 50, 900, 8000, [5] * 400 + list(range(6, 500)), 0.0),     # 400 nearest ties, then spread ones
    (8, 100, 50, 800, 8000, list(range(6, 500)) + [900] * 500, 0.0),   # spread ones, then 400 ties
    (9, 100, 50, 500, 4000, [-1.5, -0.0, 0.0, 2.0], 0.0),
])
def test_ties_beyond_a_pass_keep_the_order(gpu_ctx, seed, L, K, m, ids, distances, copies):
    c = case(seed, 16, L, m, ids, distances, copies)
    got = gpu_ctx.join_merge_check(L, K, *c)
    ref = _serial(c, L, K)
    for name, g, r in zip(("pool distances", "pool ids", "L", "radius", "found"), got, ref):
        assert np.array_equal(np.asarray(g).view(np.uint32), np.asarray(r).view(np.uint32)), name
