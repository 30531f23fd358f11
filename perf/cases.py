"""The measured work of the library: what its users run, over the sizes they run it at.

Every case is one call (or the call sequence) a program makes through
``kgraph_b200.capi.Context``: graph-walk searches, exact brute force, NN-descent
builds and reverse-edge completion.  Data follow the benchmark's generators
(uniform [0,1); non-negative integer mixtures with centres in [0,128) and
standard deviation 20; unit-norm mixtures).

A search starts from an index the program already has.  A built index differs
from run to run (the local join's threads insert in any order), so the searched
index is made here: the exact nearest neighbours of every row, completed with
reverse edges, which is what a converged build with reverse=-1 leaves.
"""
import ctypes as C
import math

import numpy as np
import torch

from kgraph_b200 import capi

DEV = "cuda"


def listed():
    return [
        # one interactive lookup: Python caller, host arrays, the package's P
        dict(name="search one query", path="search", data="uniform", n=100_000, d=16, metric="euclidean",
             nq=1, K=10, P=100, M=25, init=0, filter="fp32", mixed=False, host=True),
        # the small benchmark configuration: 1,000 uniform queries from host arrays
        dict(name="search 1k uniform", path="search", data="uniform", n=100_000, d=16, metric="euclidean",
             nq=1000, K=10, P=100, M=25, init=0, filter="fp32", mixed=False, host=True),
        # the headline data set from random seeds: P=1000 is what recall@10 0.95 takes there
        dict(name="search 10k plain", path="search", data="mixture", n=1_000_000, d=128, metric="euclidean",
             nq=10_000, K=10, P=1000, M=40, init=0, filter="fp32", mixed=False, host=False),
        # the same with user-provided starting points, at the P that suffices with good ones
        dict(name="search 10k seeded", path="search", data="mixture", n=1_000_000, d=128, metric="euclidean",
             nq=10_000, K=10, P=5, M=40, init=3, filter="fp32", mixed=False, host=False),
        # one large batch in which every query has its own K and P
        dict(name="search 100k mixed", path="search", data="mixture", n=1_000_000, d=128, metric="euclidean",
             nq=100_000, K=100, P=200, M=40, init=0, filter="fp32", mixed=True, host=False),
        # the precision configuration's search: angular with the BF16 distance filter; ragged sizes
        dict(name="search angular bf16", path="search", data="sphere", n=199_999, d=100, metric="angular",
             nq=9_973, K=10, P=700, M=40, init=0, filter="bf16", mixed=False, host=False),
        # learned entry seeds and the walk in one call
        dict(name="router search", path="router", data="mixture", n=200_000, d=128, metric="euclidean",
             nq=10_000, K=10, P=30, M=40),
        # exact k-NN, the ground truth of a recall measurement
        dict(name="brute force 10k", path="brute", data="mixture", n=1_000_000, d=128, metric="euclidean",
             nq=10_000, K=10, host=False),
        # the small benchmark configuration's build
        dict(name="build 100k uniform", path="build", data="uniform", n=100_000, d=16, metric="euclidean",
             K=25, L=50, S=10, join="auto"),
        # the headline build
        dict(name="build 1M mixture", path="build", data="mixture", n=1_000_000, d=128, metric="euclidean",
             K=50, L=100, S=12, join="auto"),
        # the precision configuration's build: angular, local join on BF16 tiles
        dict(name="build angular bf16", path="build", data="sphere", n=200_000, d=96, metric="angular",
             K=50, L=100, S=12, join="bf16"),
        # an index loaded without reverse edges and completed (the last stage of a build with reverse=-1)
        dict(name="reverse 1M", path="reverse", data="mixture", n=1_000_000, d=128, metric="euclidean", M=40),
    ]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choices(["search", "router", "brute", "build", "reverse"], [9, 1, 3, 5, 2])[0]
    data = "mixture" if path in ("router", "reverse") else rng.choice(["uniform", "mixture", "sphere"])
    # distances between all rows make the uniform and unit-norm indexes: fewer rows there
    c = dict(path=path, data=data, n=log_uniform(rng, 20_000, 1_000_000 if data == "mixture" else 200_000),
             d=rng.randint(8, 32) if data == "uniform" else rng.choice([rng.randint(33, 128), 64, 96, 128]),
             metric="angular" if data == "sphere" else rng.choice(["euclidean", "euclidean", "l2sqr"]))
    if path == "reverse":
        return dict(c, M=rng.randint(10, 50))
    if path == "router":
        return dict(c, nq=log_uniform(rng, 100, 10_000), K=10, P=rng.randint(10, 50), M=40)
    if path == "brute":
        K = rng.choice([1, 10, rng.randint(2, 100)])
        return dict(c, nq=log_uniform(rng, 1, 10_000 if K <= 10 else min(10_000, 3_000_000_000 // c["n"])), K=K,
                    host=rng.random() < 0.3)
    if path == "build":
        c["n"] = min(c["n"], 700_000)
        L = rng.choice([50, 100, rng.randint(40, 120)])
        return dict(c, K=rng.choice([25, L // 2, rng.randint(10, 40)]), L=L, S=rng.randint(8, 14),
                    join="bf16" if data == "sphere" and rng.random() < 0.5 else "auto")
    nq = log_uniform(rng, 1, 50_000)
    c.update(nq=nq, K=rng.choice([1, 10, 25, rng.randint(2, 100)]), M=rng.randint(20, 50), init=0,
             P=log_uniform(rng, 20, min(1000, 5_000_000 // nq)),
             filter=rng.choice(["fp32", "fp32", "bf16", "fp8"]), mixed=False, host=rng.random() < 0.5)
    if not c["host"] and rng.random() < 0.3:
        c.update(init=3, K=max(c["K"], 4), P=rng.randint(3, 60))
    elif not c["host"] and rng.random() < 0.3:
        c.update(mixed=True, K=max(c["K"], 10), P=max(c["P"], 40))
    return c


def make_data(case, seed, rows):
    """Base rows and `rows` more of the case's distribution, made on the GPU from the seed."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n, d = case["n"], case["d"]
    total = n + rows
    if case["data"] == "uniform":
        x = torch.rand(total, d, device=DEV, generator=g)
        return x[:n].contiguous(), x[n:].contiguous(), None
    if case["data"] == "mixture":
        centres = clusters(case)
        c = torch.rand(centres, d, device=DEV, generator=g) * 128
        lab = torch.randint(0, centres, (total,), device=DEV, generator=g)
        x = torch.randn(total, d, device=DEV, generator=g).mul_(20).add_(c[lab]).clamp_(min=0).round_()
        return x[:n].contiguous(), x[n:].contiguous(), lab[:n]
    c = torch.nn.functional.normalize(torch.randn(1000, d, device=DEV, generator=g), dim=1)
    lab = torch.randint(0, 1000, (total,), device=DEV, generator=g)
    x = torch.nn.functional.normalize(torch.randn(total, d, device=DEV, generator=g).mul_(0.3).add_(c[lab]), dim=1)
    return x[:n].contiguous(), x[n:].contiguous(), None


def clusters(case):
    """Components of the integer mixture, never fewer than 1,000 rows each: 256 at a million rows, and
    64 where a graph is built (of 256, now and then a node of one build is cut off from its own)."""
    return max(4, min(64 if case["path"] == "build" else 256, case["n"] // 1000))


def distances(case, q, x):
    """All distances of q's rows to x's in their type, by the case's metric."""
    dot = q @ x.transpose(-1, -2)
    if case["metric"] == "angular":
        return -dot / (q.norm(dim=-1)[..., :, None] * x.norm(dim=-1)[..., None, :])
    full = (q * q).sum(-1)[..., :, None] + (x * x).sum(-1)[..., None, :] - 2 * dot
    return full if case["metric"] == "l2sqr" else full / 2


def neighbours(case, x, labels, k, dtype):
    """Each row's k nearest others (ids, distances), ascending.  A mixture's components lie far
    apart, so its neighbours are looked for in the row's own component."""
    n = x.shape[0]
    ids = torch.empty(n, k, dtype=torch.int32, device=DEV)
    dist = torch.empty(n, k, dtype=dtype, device=DEV)
    if labels is None:
        groups = [None]
    else:
        order = torch.argsort(labels, stable=True)
        groups = torch.split(order, torch.bincount(labels, minlength=clusters(case)).tolist())
    for grp in groups:
        y = (x if grp is None else x[grp]).to(dtype)
        step = max(1, (1 << 29) // y.shape[0])
        for a in range(0, y.shape[0], step):
            dd = distances(case, y[a:a + step], y)
            at = torch.arange(dd.shape[0], device=DEV)
            dd[at, at + a] = math.inf
            v, i = torch.topk(dd, k, dim=1, largest=False)
            rows = at + a if grp is None else grp[a:a + step]
            ids[rows] = (i if grp is None else grp[i]).to(torch.int32)
            dist[rows] = v
    return ids, dist


def ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def import_graph(ctx, offsets, ids, dists, M):
    ctx._check(ctx.L.kg_graph_import(ctx.h, M.numel(), ptr(offsets), ptr(ids), ptr(dists), ptr(M)))


def make_index(case, x, labels, ctx):
    """The searched index: each row's M nearest, completed with reverse edges."""
    offsets, ids, dists, M = forward_graph(case, x, labels)
    torch.cuda.synchronize()
    import_graph(ctx, offsets, ids, dists, M)
    ctx.reverse(-1)


def forward_graph(case, x, labels):
    n, k = case["n"], case["M"]
    ids, dists = neighbours(case, x, labels, k, torch.float32)
    return (torch.arange(0, n * k + 1, k, device=DEV, dtype=torch.int64), ids,
            dists, torch.full((n,), k, dtype=torch.int32, device=DEV))


def prepare(case, seed):
    capi.set_verbosity(0)   # no progress lines from the library
    s = dict(case=case, ctx=capi.Context(0))
    ctx, path = s["ctx"], case["path"]
    x, q, labels = make_data(case, seed, case.get("nq", 0) + (20_000 if path == "router" else 0))
    torch.cuda.synchronize()
    ctx.set_data(x, case["metric"])
    if path == "build":
        ctx.set_join_precision(case["join"])
        s["offsets"] = torch.zeros(case["n"] + 1, dtype=torch.int64, device=DEV)
        s["ids"] = torch.zeros(case["n"], case["L"], dtype=torch.int32, device=DEV)
        s["dists"] = torch.zeros(case["n"], case["L"], device=DEV)
        torch.cuda.synchronize()
        return s
    if path == "reverse":
        s["graph"] = forward_graph(case, x, labels)
        n, E = case["n"], 2 * case["n"] * case["M"]   # room for every edge and its reverse
        s["out"] = {"offsets": torch.zeros(n + 1, dtype=torch.int64, device=DEV),
                    "ids": torch.zeros(E, dtype=torch.int32, device=DEV),
                    "dists": torch.zeros(E, device=DEV),
                    "M": torch.zeros(n, dtype=torch.int32, device=DEV)}
        torch.cuda.synchronize()
        return s
    if path != "brute":
        make_index(case, x, labels, ctx)
    nq, K = case["nq"], case["K"]
    if path == "router":
        ctx.router_train(q[nq:].cpu().numpy(), clusters=256, entries=8, label_P=500)
        q = q[:nq].contiguous()
    if path == "search":
        ctx.set_search_precision(case["filter"])
        s["params"] = capi.SearchParams(K, 0, case["P"], 10, 1, 1e30, 1998, case["init"])
        g = torch.Generator(device=DEV).manual_seed(seed + 1)
        if case["init"]:   # starting points as a router finds them: rows of the query's neighbourhood
            sample = torch.randperm(case["n"], device=DEV, generator=g)[:8192]
            near = torch.topk(distances(case, q, x[sample]), case["init"], dim=1, largest=False).indices
            s["starts"] = sample[near].to(torch.int32)
        if case["mixed"]:
            def pick(v):
                return torch.tensor(v, dtype=torch.int32, device=DEV)[torch.randint(0, 3, (nq,), device=DEV, generator=g)]
            s["Kq"], s["Pq"] = pick([1, K // 10, K]), pick([case["P"] // 4, case["P"] // 2, case["P"]])
    elif path == "router":
        s["params"] = capi.SearchParams(K, 0, case["P"], 10, 1, 1e30, 1998, 3)
    else:
        s["params"] = capi.SearchParams(K, 0, 100, 10, 1, 1e30, 1998, 0)
    if case.get("host"):
        s["queries"] = q.cpu().numpy()
        return s
    s["queries"] = q
    s["ids"] = torch.zeros(nq, K, dtype=torch.int32, device=DEV)
    s["dists"] = torch.zeros(nq, K, device=DEV)
    s["counts"] = torch.zeros(nq, dtype=torch.int32, device=DEV)
    s["costs"] = torch.zeros(nq, device=DEV)
    torch.cuda.synchronize()
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    path = case["path"]
    if path == "build":
        ctx.build(iterations=30, K=case["K"], L=case["L"], S=case["S"], R=100)
        ctx._check(ctx.L.kg_graph_export(ctx.h, ptr(s["offsets"]), ptr(s["ids"]), ptr(s["dists"]), None))
        # ids and M differ between two builds (one neighbour more or less moves a row's rest along);
        # the sorted distances hardly do
        return {"offsets": s["offsets"], "dists": s["dists"]}
    if path == "reverse":
        import_graph(ctx, *s["graph"])
        ctx.reverse(-1)
        ctx._check(ctx.L.kg_graph_export(ctx.h, *(ptr(s["out"][k]) for k in ("offsets", "ids", "dists", "M"))))
        return s["out"]
    if case.get("host"):
        ids, dists, counts, costs = ctx.search(s["queries"], K=case["K"], P=case.get("P", 100))
        return {"ids": ids, "dists": dists, "counts": counts, "costs": costs}
    q, K = s["queries"], case["K"]
    outs = (ptr(s["ids"]), ptr(s["dists"]), ptr(s["counts"]), ptr(s["costs"]))
    if path == "router":
        ctx.router_search_raw(ptr(q), q.shape[0], q.stride(0) * 4, s["params"], K, *outs)
    else:
        if "starts" in s:   # the output ids are the input of the starting points
            s["ids"][:, :case["init"]] = s["starts"]
            torch.cuda.current_stream().synchronize()   # the library works on its own stream
        ctx.search_raw(ptr(q), q.shape[0], q.stride(0) * 4, s["params"], ptr(s.get("Kq")), ptr(s.get("Pq")), K, *outs)
    return {k: s[k] for k in ("ids", "dists", "counts", "costs")}


def work(case):
    n, d = case["n"], case["d"]
    if case["path"] == "build":
        # the join's pairs per node until the lists stop changing, as the three generators give them
        pairs = {"uniform": 1900, "mixture": 5000, "sphere": 11000}[case["data"]] * case["L"] / (
            50 if case["data"] == "uniform" else 100)
        return {"bytes": n * (4 * d + 8 * case["L"]), "flops": 2 * d * pairs * n}
    if case["path"] == "reverse":
        return {"bytes": 3 * 8 * n * case["M"], "flops": 0}
    nq, K = case["nq"], case["K"]
    io = nq * (4 * d + 8 * K + 8)
    if case["path"] == "brute":
        return {"bytes": 4 * n * d + io, "flops": 2.0 * n * nq * d}
    # a walk: every entry of its final list is expanded once, and so are those it came by; each
    # neighbour is read, and its row where the walk has not met it before
    K, P = (0.37 * K, 0.58 * case["P"]) if case.get("mixed") else (K, case["P"])
    adjacency = (K + P + 20) * 1.6 * case["M"]
    rows = {"uniform": 0.6 * adjacency, "mixture": min(0.67 * adjacency, P + 4000), "sphere": 0.8 * adjacency}
    rows = min(n, rows[case["data"]])
    return {"bytes": io + nq * (rows * (4 * d + 4) + 4 * adjacency), "flops": nq * rows * 2 * d}


def exact(case, seed):
    """The exact neighbours' distances in 64 bits: what brute force returns, and what a build comes
    close to.  Ids of equal distances and a walk's results have no such value."""
    if case["path"] == "build":
        x, _, labels = make_data(case, seed, 0)
        n, L = case["n"], case["L"]
        return {"offsets": None, "dists": neighbours(case, x, labels, L, torch.float64)[1]}
    if case["path"] != "brute":
        return None
    x, q, _ = make_data(case, seed, case["nq"])
    x, q = x.double(), q.double()
    step = max(1, (1 << 29) // x.shape[0])
    best = [torch.topk(distances(case, q[a:a + step], x), case["K"], dim=1, largest=False).values
            for a in range(0, q.shape[0], step)]
    return {"ids": None, "dists": torch.cat(best), "counts": None, "costs": None}
