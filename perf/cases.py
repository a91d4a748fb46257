"""The calls whose speed this library is judged by, one dict per case.

    call   graph                 what it stands for
    bfs    er / rmat / grid      distance rows from k sources (gu_bfs, AUTO)
    reach  dag                   reachable counts without rows (a reachability query)
    dag    dag                   reachable-set size of every vertex (gu_dag_reach)
    bc     er / rmat             FP64 Brandes betweenness from k sources
    sigma  rmat                  shortest-path counts with distance rows
    lbs    grid / pareto / zero  load-balanced search over an array of work counts
    many   rmat + dag            a set of requests on several graphs in one launch
    diam   grid                  largest distance from k sources (drawn cases)

Graphs are made on the GPU from the seed alone and handed to the library as host
CSR arrays, as a program that loads its graph does; sources are device arrays.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "graph-utils_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gu  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # exact analysis of a small social graph: BFS from every vertex (C1 of the benchmark set)
        {"name": "bfs_er198_all", "call": "bfs", "graph": "er", "n": 198, "m": 2742, "k": 198, "pad": 0},
        # one query on a resident graph: a single source, where the latency of the levels counts
        {"name": "bfs_rmat17_one", "call": "bfs", "graph": "rmat", "scale": 17, "ef": 16, "k": 1, "pad": 0},
        # an ordinary request: 150 sources on a graph of 16 K vertices (the tests' own size)
        {"name": "bfs_rmat14_150", "call": "bfs", "graph": "rmat", "scale": 14, "ef": 16, "k": 150, "pad": 0},
        # the headline benchmark: R-MAT scale 20, 512 sources
        {"name": "bfs_rmat20_512", "call": "bfs", "graph": "rmat", "scale": 20, "ef": 16, "k": 512, "pad": 0},
        # road-network-like: high diameter, low degree, 256 sources (C4)
        {"name": "bfs_grid2048_256", "call": "bfs", "graph": "grid", "rows": 2048, "cols": 2048, "k": 256, "pad": 0},
        # reachability query on a dependency graph, odd sizes, no rows
        {"name": "reach_dag200003_200", "call": "reach", "graph": "dag", "n": 200003, "deg": 8, "k": 200},
        # the whole closure of a dependency graph, as set sizes
        {"name": "dag65536_all", "call": "dag", "graph": "dag", "n": 65536, "deg": 8},
        # exact betweenness of a small social graph (C1)
        {"name": "bc_er198_all", "call": "bc", "graph": "er", "n": 198, "m": 2742, "k": 198, "batch": 0},
        # sampled betweenness of a large graph, the widest pass (C3)
        {"name": "bc_rmat18_1024", "call": "bc", "graph": "rmat", "scale": 18, "ef": 16, "k": 1024, "batch": 1024},
        # shortest-path counts and distances as rows
        {"name": "sigma_rmat16_200", "call": "sigma", "graph": "rmat", "scale": 16, "ef": 16, "k": 200},
        # edge extraction of a whole mesh: the degree array of a 2048 x 2048 grid (C4)
        {"name": "lbs_grid_4m", "call": "lbs", "graph": "grid", "n": 2048 * 2048},
        # a serving batch: BFS and reachability requests on small resident graphs
        {"name": "many_24", "call": "many", "requests": 24, "kmax": 256, "smin": 12, "smax": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["bfs", "bfs", "bfs", "bfs", "reach", "dag", "bc", "bc", "sigma", "lbs", "lbs", "many", "diam"])
    if call in ("bfs", "diam"):
        graph = rng.choice(["er", "rmat", "rmat", "grid"]) if call == "bfs" else "grid"
        c = {"call": call, "graph": graph, "k": _log(rng, 1, 512)}
        if graph == "er":  # from all-pairs analysis of a few hundred vertices up
            c["n"] = _log(rng, 150, 300000)
            c["m"] = c["n"] * rng.randint(10, 14)
            c["k"] = min(c["k"], c["n"])
        elif graph == "rmat":
            c["scale"] = rng.randint(10, 20)
            c["ef"] = rng.randint(4, 16)
        else:
            c["rows"], c["cols"] = _log(rng, 48, 2048), _log(rng, 48, 2048)
            c["k"] = min(c["k"], 256)
        if call == "bfs":
            c["pad"] = rng.choice([0, 0, 0, 5])  # rows inside a wider buffer
        return c
    if call == "reach":
        return {"call": call, "graph": "dag", "n": _log(rng, 5000, 200003), "deg": rng.randint(4, 10), "k": _log(rng, 1, 256)}
    if call == "dag":
        return {"call": call, "graph": "dag", "n": _log(rng, 3000, 65536), "deg": rng.randint(4, 8)}
    if call == "bc":
        if rng.random() < 0.5:
            n = _log(rng, 150, 4000)
            return {"call": call, "graph": "er", "n": n, "m": n * rng.randint(8, 14), "k": min(n, _log(rng, 32, 1024)), "batch": 0}
        return {"call": call, "graph": "rmat", "scale": rng.randint(10, 18), "ef": rng.randint(4, 16), "k": _log(rng, 16, 1024),
                "batch": rng.choice([0, 64, 128, 256, 512, 1024])}
    if call == "sigma":
        return {"call": call, "graph": "rmat", "scale": rng.randint(10, 17), "ef": rng.randint(4, 16), "k": _log(rng, 8, 256)}
    if call == "lbs":
        return {"call": call, "graph": rng.choice(["grid", "pareto", "zero"]), "n": _log(rng, 1000, 4194304)}
    return {"call": "many", "requests": rng.randint(2, 32), "kmax": _log(rng, 8, 256), "smin": 11, "smax": rng.randint(12, 16)}


# ---- inputs -------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _csr(n, u, v, symmetric):
    """Sorted, deduplicated CSR without self-loops (int32 device tensors)."""
    if symmetric:
        u, v = torch.cat([u, v]), torch.cat([v, u])
    key = torch.unique((u * n + v)[u != v])
    src = torch.div(key, n, rounding_mode="floor")
    R = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    R[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    return R.to(torch.int32), (key - src * n).to(torch.int32)


def _rmat(scale, ef, g):
    """R-MAT with (a, b, c) = (0.57, 0.19, 0.19), vertices relabelled at random."""
    n, m = 1 << scale, ef << scale
    u = torch.zeros(m, dtype=torch.int64, device=DEV)
    v = torch.zeros(m, dtype=torch.int64, device=DEV)
    for _ in range(scale):
        p = torch.rand(m, generator=g, device=DEV)
        u = 2 * u + (p >= 0.76)
        v = 2 * v + (((p >= 0.57) & (p < 0.76)) | (p >= 0.95))
    perm = torch.randperm(n, generator=g, device=DEV)
    return n, *_csr(n, perm[u], perm[v], True)


def _er(n, m, g):
    u = torch.randint(0, n, (m,), generator=g, device=DEV)
    v = torch.randint(0, n, (m,), generator=g, device=DEV)
    return n, *_csr(n, u, v, True)


def _grid(rows, cols, g):
    """4-neighbour grid, each edge deleted with probability 0.05."""
    ids = torch.arange(rows * cols, device=DEV).reshape(rows, cols)
    u = torch.cat([ids[:, :-1].reshape(-1), ids[:-1].reshape(-1)])
    v = torch.cat([ids[:, 1:].reshape(-1), ids[1:].reshape(-1)])
    keep = torch.rand(u.numel(), generator=g, device=DEV) >= 0.05
    return rows * cols, *_csr(rows * cols, u[keep], v[keep], True)


def _dag(n, m, g):
    """m random edges, each from the earlier to the later vertex of a random order."""
    a = torch.randint(0, n, (m,), generator=g, device=DEV)
    b = torch.randint(0, n, (m,), generator=g, device=DEV)
    perm = torch.randperm(n, generator=g, device=DEV)
    return n, *_csr(n, perm[torch.minimum(a, b)], perm[torch.maximum(a, b)], False)


def _arrays(case, g):
    if case["graph"] == "rmat":
        return _rmat(case["scale"], case["ef"], g)
    if case["graph"] == "er":
        return _er(case["n"], case["m"], g)
    if case["graph"] == "grid":
        return _grid(case["rows"], case["cols"], g)
    return _dag(case["n"], case["n"] * case["deg"], g)


def _graph(n, R, C, directed):
    return gu.Graph(gu.HostGraph(R.cpu().numpy(), C.cpu().numpy(), n, directed))


def _sources(n, R, k, g):
    """k distinct vertices at random; vertices without out-edges only when no others are left."""
    p = torch.randperm(n, generator=g, device=DEV)
    has = (R[1:] > R[:-1])[p]
    return torch.cat([p[has], p[~has]])[:k].to(torch.int32).contiguous()


def _counts(case, g):
    """Work counts per item: degrees of a mesh, of a skewed graph, or of a sparse frontier."""
    n = case["n"]
    if case["graph"] == "grid":
        return (torch.rand((n, 4), generator=g, device=DEV) >= 0.05).sum(1).to(torch.int32)
    if case["graph"] == "pareto":
        p = torch.rand(n, generator=g, device=DEV).clamp_min(1e-7)
        return (p ** -0.7).to(torch.int32).clamp_max(200000)
    on = torch.rand(n, generator=g, device=DEV) < 0.1
    return torch.where(on, torch.randint(1, 40, (n,), generator=g, device=DEV), 0).to(torch.int32)


def prepare(case, seed):
    g = _gen(seed)
    call = case["call"]
    if call == "lbs":
        counts = _counts(case, g)
        cap = {"grid": 4 * case["n"], "pareto": 6 * case["n"] + 400000, "zero": 4 * case["n"]}[case["graph"]]
        return {"case": case, "counts": counts, "scanned": torch.empty_like(counts),
                "result": torch.zeros(cap, dtype=torch.int32, device=DEV)}
    if call == "many":
        graphs, reqs = [], []
        for i in range(6):
            scale = case["smin"] + i % (case["smax"] - case["smin"] + 1)
            graphs.append((_rmat(scale, 8 if i % 2 else 16, g), False))
        for i in range(2):
            n = (1 << case["smax"]) - 1000 * i
            graphs.append((_dag(n, 8 * n, g), True))
        graphs = [(_graph(*a, d), a[1], d) for a, d in graphs]
        sizes = random.Random(case["requests"] * 1000 + case["kmax"])
        for i in range(case["requests"]):
            k = sizes.randint(1, case["kmax"])
            gr, R, directed = graphs[i % len(graphs)]
            s = _sources(gr.n, R, k, g)
            if directed:  # reachability on the dependency graphs, rows elsewhere
                reqs.append((gr, s, None, torch.empty(k, dtype=torch.int64, device=DEV)))
            else:
                reqs.append((gr, s, torch.empty((k, gr.n), dtype=torch.int32, device=DEV), None))
        return {"case": case, "reqs": reqs}
    n, R, C = _arrays(case, g)
    gr = _graph(n, R, C, case["graph"] == "dag")
    st = {"case": case, "g": gr}
    if call == "dag":
        st["counts"] = torch.empty(n, dtype=torch.int64, device=DEV)
        return st
    k = min(case["k"], n)
    st["s"] = _sources(n, R, k, g)
    if call == "bfs":
        st["ld"] = n + case["pad"]
        st["dist"] = torch.zeros((k, st["ld"]), dtype=torch.int32, device=DEV)
    elif call == "reach":
        st["counts"] = torch.empty(k, dtype=torch.int64, device=DEV)
    elif call == "bc":
        st["bc"] = torch.empty(n, dtype=torch.float64, device=DEV)
    elif call == "sigma":
        st["sigma"] = torch.empty((k, n), dtype=torch.int64, device=DEV)
        st["dist"] = torch.empty((k, n), dtype=torch.int32, device=DEV)
    return st


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "bfs":
        return state["g"].bfs(state["s"], state["dist"], ld=state["ld"])
    if call == "reach":
        state["g"].reach(state["s"], state["counts"])
        return state["counts"]
    if call == "dag":
        total = state["g"].dag_reach(state["counts"])
        return [state["counts"], total]
    if call == "bc":
        return state["g"].bc(state["s"], state["bc"], batch=case["batch"])
    if call == "sigma":
        state["g"].sigma(state["s"], state["sigma"], dist_dev=state["dist"])
        return [state["sigma"], state["dist"]]
    if call == "diam":
        # every source's distances count towards it; the rows themselves are not asked for
        return state["g"].diameter(state["s"])
    if call == "lbs":
        total = gu.lbs(state["counts"], state["scanned"], state["result"])
        return [state["scanned"], state["result"], total]
    gu.bfs_many(state["reqs"])
    return [d if d is not None else r for _, _, d, r in state["reqs"]]


# ---- what a pass cannot do without ------------------------------------------------------
def _size(case):
    """(vertices, CSR entries) of the case's graph, before duplicates are dropped."""
    if case["graph"] == "rmat":
        return 1 << case["scale"], 2 * case["ef"] << case["scale"]
    if case["graph"] == "er":
        return case["n"], 2 * case["m"]
    if case["graph"] == "grid":
        n = case["rows"] * case["cols"]
        return n, int(3.8 * n)
    return case["n"], case["n"] * case["deg"]


def work(case):
    call = case["call"]
    if call == "lbs":
        n = case["n"]
        total = {"grid": 3.8, "pareto": 2.8, "zero": 2.0}[case["graph"]] * n
        return {"bytes": 8 * n + 4 * total, "flops": 0}
    if call == "many":
        b = 0
        for i in range(case["requests"]):
            j = i % 8
            n = 1 << (case["smin"] + j % (case["smax"] - case["smin"] + 1) if j < 6 else case["smax"])
            b += 4 * n * (17 if j % 2 else 33) + (4 * n * case["kmax"] // 2 if j < 6 else 0)
        return {"bytes": b, "flops": 0}
    n, m = _size(case)
    csr = 4 * (n + 1) + 4 * m
    if call == "dag":
        return {"bytes": csr + 8 * n, "flops": 0}
    k = min(case["k"], n)
    if call == "bc":
        # one addition per edge and source on the way out and one on the way back
        return {"bytes": csr + 8 * n, "flops": 1.0 * m * k}
    if call == "sigma":
        return {"bytes": csr + 12 * n * k, "flops": 0}
    return {"bytes": csr + (4 * n * k if call == "bfs" else 8 * k), "flops": 0}


# ---- 64-bit values of the floating-point results --------------------------------------------
def exact(case, seed):
    """Betweenness by Brandes' recurrences on dense float64 blocks of sources; the
    other calls return whole numbers."""
    if case["call"] != "bc":
        return None
    g = _gen(seed)
    n, R, C = _arrays(case, g)
    s = _sources(n, R, min(case["k"], n), g).long()
    A = torch.sparse_csr_tensor(R.long(), C.long(), torch.ones(C.numel(), dtype=torch.float64, device=DEV), (n, n))
    bc = torch.zeros(n, dtype=torch.float64, device=DEV)
    for b in range(0, s.numel(), 128):
        sb = s[b:b + 128]
        cols = torch.arange(sb.numel(), device=DEV)
        level = torch.full((n, sb.numel()), -1, dtype=torch.int32, device=DEV)
        sigma = torch.zeros((n, sb.numel()), dtype=torch.float64, device=DEV)
        level[sb, cols] = 0
        sigma[sb, cols] = 1.0
        L = 0
        while True:  # forward: path counts level by level
            x = A @ torch.where(level == L, sigma, 0.0)
            new = (x > 0) & (level < 0)
            if not bool(new.any()):
                break
            L += 1
            level[new] = L
            sigma = torch.where(new, x, sigma)
        delta = torch.zeros_like(sigma)
        for lv in range(L - 1, 0, -1):  # backward: dependencies
            y = A @ torch.where(level == lv + 1, (1.0 + delta) / sigma.clamp_min(1.0), 0.0)
            delta = torch.where(level == lv, sigma * y, delta)
        bc += delta.sum(1)
    return bc
