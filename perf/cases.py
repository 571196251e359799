"""What the framework is measured on: its graph algorithms through ``DeviceGraph``, on
seeded synthetic graphs that are made on the GPU.

A case names an algorithm and a graph. A user's program uploads a graph once and keeps the
``DeviceGraph`` (and the device arrays that results go to); a pass is one call of the
algorithm on it. The graphs have the shapes of the benchmark workloads: R-MAT (skewed
degrees), uniformly random (ER), 2-D grids (high diameter) and planted partitions, from a
few thousand edges to the largest workload of each algorithm, vertex counts that are no
power of two among them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from starplat_b200.device import DeviceGraph

DEV = "cuda"
INT_MAX = 2**31 - 1


def listed():
    return [
        # Triangle counting. The small one stands for calls on small graphs, where the
        # launches and the wait for the count decide; R-MAT 16 is the usual benchmark
        # graph; R-MAT 20 the largest that the centrality workloads use.
        {"name": "tc_rmat12", "algo": "tc", "graph": "rmat", "n": 4096, "ef": 8, "directed": False},
        {"name": "tc_rmat16", "algo": "tc", "graph": "rmat", "n": 65536, "ef": 16, "directed": False},
        {"name": "tc_rmat20", "algo": "tc", "graph": "rmat", "n": 1 << 20, "ef": 16, "directed": False},
        # Triangles of every vertex (the clustering coefficient's input), between the two.
        {"name": "clustering_rmat18", "algo": "clustering", "graph": "rmat", "n": 1 << 18, "ef": 16,
         "directed": False},
        # PageRank until convergence: a middle-sized graph without hubs whose vertex count
        # is odd, and the headline workload.
        {"name": "pagerank_er100003", "algo": "pagerank", "graph": "er", "n": 100003, "ef": 16, "directed": True},
        {"name": "pagerank_rmat22", "algo": "pagerank", "graph": "rmat", "n": 1 << 22, "ef": 16, "directed": True},
        # Shortest paths from one source: the skewed low-diameter graph and the grid (road
        # networks behave like it).
        {"name": "sssp_rmat23", "algo": "sssp", "graph": "rmat", "n": 1 << 23, "ef": 16, "directed": True,
         "wmax": 100},
        {"name": "sssp_grid4096", "algo": "sssp", "graph": "grid", "rows": 4096, "cols": 4096, "wmax": 1000},
        # Betweenness: many sources on one graph, and many small graphs in one call.
        {"name": "bc_rmat20", "algo": "bc", "graph": "rmat", "n": 1 << 20, "ef": 16, "directed": False,
         "sources": 256},
        {"name": "bc_graphs_er1000", "algo": "bc_graphs", "graph": "ers", "graphs": 1000, "nmin": 1000,
         "nmax": 50000, "dmin": 8, "dmax": 32, "sources": 16},
        # Communities of a social-network-like planted partition.
        {"name": "louvain_sbm1m", "algo": "louvain", "graph": "sbm", "n": 1 << 20, "blocks": 256, "degree": 32,
         "weights": "none"},
        # A graph that changes: a batch of edge updates, ranks brought up to date, the
        # batch undone, ranks again (the rebuilt CSR's plans are part of it).
        {"name": "pagerank_update_rmat20", "algo": "pagerank_update", "graph": "rmat", "n": 1 << 20, "ef": 16,
         "directed": True, "batch": 4096},
    ]


def _spread(rng, lo, hi):
    """An integer of [lo, hi], spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    algo = rng.choice(["tc", "tc", "clustering", "pagerank", "pagerank", "sssp", "sssp", "bc", "bc_graphs", "louvain",
                       "pagerank_update"])
    c = {"algo": algo}
    if algo in ("tc", "clustering"):
        c["graph"] = rng.choice(["rmat", "rmat", "er"])
        c["directed"] = rng.random() < 0.25
        c["ef"] = rng.randint(4, 16)
        c["n"] = _spread(rng, 1000, 1 << 15 if c["directed"] else 1 << 20 if algo == "tc" else 1 << 18)
    elif algo == "pagerank":
        c["graph"] = rng.choice(["rmat", "er"])
        c["directed"] = rng.random() < 0.75
        c["n"] = _spread(rng, 1000, 1 << 21)
        c["ef"] = rng.randint(4, 16)
    elif algo == "sssp":
        c["graph"] = rng.choice(["rmat", "er", "grid"])
        c["wmax"] = rng.choice([1, 10, 100, 1000])
        if c["graph"] == "grid":
            c["rows"], c["cols"] = _spread(rng, 20, 4096), _spread(rng, 20, 4096)
        else:
            c["directed"] = rng.random() < 0.5
            c["n"] = _spread(rng, 1000, 1 << 22)
            c["ef"] = rng.randint(4, 16)
    elif algo == "bc":
        c["graph"] = rng.choice(["rmat", "er"])
        c["directed"] = rng.random() < 0.25
        c["n"] = _spread(rng, 1000, 1 << 19)
        c["ef"] = rng.randint(4, 16)
        c["sources"] = rng.choice([1, 7, 16, 33, 64, 100, 256])
    elif algo == "bc_graphs":
        c["graph"] = "ers"
        c["graphs"] = _spread(rng, 10, 600)
        c["nmin"] = _spread(rng, 200, 2000)
        c["nmax"] = _spread(rng, 4000, 50000)
        c["dmin"], c["dmax"] = 4, rng.randint(8, 32)
        c["sources"] = rng.choice([5, 16, 24, 40])
    elif algo == "louvain":
        c["graph"] = "sbm"
        c["n"] = _spread(rng, 2000, 1 << 20)
        c["blocks"] = rng.randint(8, 256)
        c["degree"] = rng.randint(8, 32)
        c["weights"] = rng.choice(["none", "whole"])
    else:
        c["graph"] = "rmat"
        c["directed"] = True
        c["n"] = _spread(rng, 5000, 1 << 20)
        c["ef"] = rng.randint(4, 16)
        c["batch"] = _spread(rng, 16, 8192)
    return c


# ------------------------------------------------------------------- graphs, on the GPU
def _csr(V, key):
    """Offsets and neighbours of sorted distinct keys src * V + dst."""
    off = torch.searchsorted(key, torch.arange(V + 1, device=DEV, dtype=torch.int64) * V).to(torch.int32)
    return off, (key % V).to(torch.int32)


def _keys(V, src, dst, both):
    """Sorted distinct keys src * V + dst without self-loops; `both`: in both directions."""
    ok = (src != dst) & (src < V) & (dst < V)
    src, dst = src[ok], dst[ok]
    key = torch.cat([src * V + dst, dst * V + src]) if both else src * V + dst
    return torch.unique(key)


def _rmat_pairs(n, pairs, gen):
    """R-MAT pairs (a, b, c, d = .57, .19, .19, .05) on the next power of two of ids."""
    src = torch.zeros(pairs, dtype=torch.int64, device=DEV)
    dst = torch.zeros(pairs, dtype=torch.int64, device=DEV)
    for _ in range(max(1, (n - 1).bit_length())):
        u = torch.rand(pairs, generator=gen, device=DEV)
        right = ((u >= 0.57) & (u < 0.76)) | (u >= 0.95)
        src.mul_(2).add_(u >= 0.76)
        dst.mul_(2).add_(right)
    return src, dst


def _sbm_pairs(n, blocks, degree, gen):
    """Planted partition: power-law block sizes, 80 % of the pairs inside a block."""
    u = torch.rand(blocks, generator=gen, device=DEV, dtype=torch.float64)
    size = (1.0 / (1.0 - 0.999 * u)).clamp(max=200.0)  # density ~ size^-2
    edge = torch.cumsum(size / size.sum(), 0) * (n - 2 * blocks)
    start = torch.cat([torch.zeros(1, device=DEV, dtype=torch.int64), edge.to(torch.int64)])
    start = start + 2 * torch.arange(blocks + 1, device=DEV)
    start[-1] = n
    m = n * degree // 2
    src = torch.randint(n, (m,), generator=gen, device=DEV)
    b = torch.searchsorted(start, src, right=True) - 1
    lo, hi = start[b], start[b + 1]
    r = torch.rand(m, generator=gen, device=DEV, dtype=torch.float64)
    inside = lo + ((hi - lo) * r).to(torch.int64).clamp(max=n)
    out = torch.randint(n, (m,), generator=gen, device=DEV)
    p = torch.rand(m, generator=gen, device=DEV)
    return src, torch.where(p < 0.8, torch.minimum(inside, hi - 1), out)


def _weights(V, src, dst, wmax, seed):
    """Weights of [1, wmax], the same in both directions of an edge."""
    lo, hi = torch.minimum(src, dst), torch.maximum(src, dst)
    h = (lo * V + hi) * 0x9E3779B1 + seed * 0x85EBCA77
    h = (h ^ (h >> 29)) * 0x2545F4914F6CDD1D
    h = (h ^ (h >> 32)) & 0x7FFFFFFF
    return (1 + h % wmax).to(torch.int32)


def _graph(case, seed):
    """The case's graph as a dict: V, key (sorted src * V + dst), off, adj, and roff, radj
    (the reverse CSR; the same tensors where every edge has its opposite)."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    kind = case["graph"]
    sym = not case.get("directed", False)
    g = {"gen": gen}
    if kind == "rmat":
        V = case["n"]
        key = _keys(V, *_rmat_pairs(V, case["ef"] * V, gen), sym)
    elif kind == "er":
        V = case["n"]
        pairs = torch.randint(V, (2, case["ef"] * V), generator=gen, device=DEV)
        key = _keys(V, pairs[0], pairs[1], sym)
    elif kind == "grid":
        R, C = case["rows"], case["cols"]
        V = R * C
        v = torch.arange(V, device=DEV, dtype=torch.int64)
        right, down = v[v % C < C - 1], v[: V - C]
        key = _keys(V, torch.cat([right, down]), torch.cat([right + 1, down + C]), True)
    elif kind == "sbm":
        V = case["n"]
        key = _keys(V, *_sbm_pairs(V, case["blocks"], case["degree"], gen), True)
    else:  # many ER graphs as one disjoint union
        r = np.random.default_rng(11)  # the sizes belong to the case, the edges to the seed
        n = np.exp(r.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["graphs"])).round().astype(np.int64)
        d = r.uniform(case["dmin"], case["dmax"], case["graphs"])
        voff = np.concatenate([[0], np.cumsum(n)])
        m = torch.from_numpy((n * d / 2).round().astype(np.int64)).to(DEV)
        V = int(voff[-1])
        base = torch.repeat_interleave(torch.from_numpy(voff[:-1].copy()).to(DEV), m)
        size = torch.repeat_interleave(torch.from_numpy(n).to(DEV), m)
        u = torch.rand((2, base.numel()), generator=gen, device=DEV, dtype=torch.float64)
        ends = torch.minimum((u * size).to(torch.int64), size - 1) + base
        key = _keys(V, ends[0], ends[1], True)
        k = case["sources"]
        g["voff"] = voff.astype(np.int32)
        g["soff"] = np.arange(0, k * (case["graphs"] + 1), k, dtype=np.int32)
        r = np.random.default_rng(seed)
        g["sources"] = np.concatenate([np.sort(r.choice(s, k, replace=False)) + b
                                       for s, b in zip(n, voff)]).astype(np.int32)
    g["V"], g["key"] = V, key
    g["off"], g["adj"] = _csr(V, key)
    if sym:
        g["roff"], g["radj"] = g["off"], g["adj"]
    else:
        g["roff"], g["radj"] = _csr(V, torch.sort((key % V) * V + key // V).values)
    if "wmax" in case:
        g["w"] = _weights(V, key // V, key % V, case["wmax"], seed)
    if case["algo"] in ("bc", "sssp"):  # sources with out-edges, as the benchmark picks them
        cand = torch.nonzero(g["off"][1:] > g["off"][:-1]).reshape(-1)
        take = min(case.get("sources", 1), cand.numel())
        pick = torch.randperm(cand.numel(), generator=gen, device=DEV)[:take]
        g["sources"] = cand[pick].sort().values.to(torch.int32).cpu().numpy()
    return g


def _ranks64(off, roff, radj, pr, iters, beta=0.0, damping=0.85):
    """PageRank in FP64 from the ranks pr: until the L1 change is at most beta, or iters."""
    V = off.numel() - 1
    deg = (off[1:] - off[:-1]).double().clamp(min=1)
    a = torch.sparse_csr_tensor(roff, radj, torch.ones(radj.numel(), dtype=torch.float64, device=DEV), (V, V))
    for _ in range(iters):
        new = (1 - damping) / V + damping * torch.mv(a, pr / deg)
        diff = (new - pr).abs().sum()
        pr = new
        if beta and float(diff) <= beta:
            break
    return pr


def _batch(case, g):
    """Half deletions of edges that are there, half additions of edges that are not."""
    V, key, gen, nb = g["V"], g["key"], g["gen"], case["batch"]
    pick = torch.randperm(key.numel(), generator=gen, device=DEV)[: min(nb // 2, key.numel())]
    gone = key[pick]
    pairs = torch.randint(V, (2, nb), generator=gen, device=DEV)
    new = _keys(V, pairs[0], pairs[1], False)
    at = torch.searchsorted(key, new).clamp(max=key.numel() - 1)
    new = new[key[at] != new]
    new = new[torch.randperm(new.numel(), generator=gen, device=DEV)[: nb - nb // 2]]
    return gone, new


# ------------------------------------------------------------------- the measured calls
def prepare(case, seed):
    g = _graph(case, seed)
    V, algo = g["V"], case["algo"]
    dg = DeviceGraph(g["off"], g["adj"], g.get("w"), g["roff"], g["radj"])
    s = {"algo": algo, "dg": dg}
    if algo == "clustering":
        s["out"] = torch.empty(V, dtype=torch.int32, device=DEV)
    elif algo == "pagerank":
        s["out"] = torch.empty(V, dtype=torch.float32, device=DEV)
    elif algo == "sssp":
        s["src"] = int(g["sources"][0])
        s["out"] = torch.empty(V, dtype=torch.int32, device=DEV)
    elif algo in ("bc", "bc_graphs"):
        s["sources"] = g["sources"]
        s["out"] = torch.empty(V, dtype=torch.float32, device=DEV)
        if algo == "bc_graphs":
            s["voff"], s["soff"] = g["voff"], g["soff"]
    elif algo == "louvain":
        s["out"] = torch.empty(V, dtype=torch.int32, device=DEV)
        s["weight"] = None
        if case["weights"] == "whole":
            s["weight"] = _weights(V, g["key"] // V, g["key"] % V, 8, seed).float()
    elif algo == "pagerank_update":
        gone, new = _batch(case, g)
        one = torch.full((V,), 1.0 / V, dtype=torch.float64, device=DEV)
        s["ranks"] = _ranks64(g["off"], g["roff"], g["radj"], one, 100, 1e-7).float()
        s["out"] = [torch.empty_like(s["ranks"]) for _ in range(2)]
        both = torch.cat([gone, new])
        s["ends"] = [(both // V).to(torch.int32).cpu().numpy(), (both % V).to(torch.int32).cpu().numpy()]
        s["types"] = ["d" * gone.numel() + "a" * new.numel(), "a" * gone.numel() + "d" * new.numel()]
    return s


def run(s):
    dg, algo = s["dg"], s["algo"]
    if algo == "tc":
        return dg.tc()
    if algo == "clustering":
        return dg.clustering_coeff(out=s["out"])
    if algo == "pagerank":
        return dg.pagerank(1e-6, 0.85, 100, out=s["out"])
    if algo == "sssp":
        return dg.sssp(s["src"], out=s["out"])[0]
    if algo == "bc":
        return dg.bc(s["sources"], out=s["out"])
    if algo == "bc_graphs":
        return dg.bc_graphs(s["voff"], s["soff"], s["sources"], out=s["out"])
    if algo == "louvain":
        return dg.louvain(s["weight"], 1e-4, community=s["out"])
    got, ranks = [], s["ranks"]
    for types, out in zip(s["types"], s["out"]):  # the batch, then its opposite
        out.copy_(ranks)
        got.append(dg.pagerank_dynamic(types, *s["ends"], None, out, 1e-6, 0.85, 100))
        ranks = out
    return got


def work(case):
    """Each input array read once and each output written once; an operation per edge (and
    source). The sizes are the nominal ones: duplicate pairs are not subtracted."""
    kind, algo = case["graph"], case["algo"]
    both = 1 if case.get("directed", False) else 2
    if kind == "grid":
        V = case["rows"] * case["cols"]
        E = 4 * V - 2 * (case["rows"] + case["cols"])
    elif kind == "sbm":
        V = case["n"]
        E = V * case["degree"]
    elif kind == "ers":
        lo, hi = case["nmin"], case["nmax"]
        V = int(case["graphs"] * (hi - lo) / math.log(hi / lo))
        E = int(V * (case["dmin"] + case["dmax"]) / 2)
    else:
        V = case["n"]
        E = both * case["ef"] * V
    csr = 4 * (V + 1) + 4 * E
    if algo == "tc":
        return {"bytes": csr + 8, "flops": E}
    if algo == "clustering":
        return {"bytes": csr + 4 * V, "flops": E}
    if algo == "pagerank":  # the reverse rows, the out-degrees, the ranks
        return {"bytes": csr + 4 * V + 4 * V, "flops": 2 * E}
    if algo == "sssp":
        return {"bytes": csr + 4 * E + 4 * V, "flops": E}
    if algo in ("bc", "bc_graphs"):
        return {"bytes": csr + 4 * V, "flops": 2 * E * case["sources"]}
    if algo == "louvain":
        return {"bytes": csr + 4 * V + (4 * E if case["weights"] == "whole" else 0), "flops": 2 * E}
    return {"bytes": 2 * (2 * csr + 4 * V + 4 * V + 4 * V + 9 * case["batch"]), "flops": 4 * E}


# ------------------------------------------------------------------- 64-bit values
def _triangles64(g):
    """(count, per-vertex counts) of v's neighbours u < v < w joined by u -> w."""
    V = g["V"]
    a = torch.zeros((V, V), dtype=torch.float64, device=DEV)
    a.view(-1)[g["key"]] = 1.0
    low, up = torch.tril(a, -1), torch.triu(a, 1)
    m = (low.T @ up) * a  # [u, w]
    per = m.sum(1) + m.sum(0) + (low * (up @ a.T)).sum(1)
    return int(m.sum().round()), per.round().to(torch.int32)


def _paths64(g, src):
    dist = torch.full((g["V"],), INT_MAX, dtype=torch.int64, device=DEV)
    dist[src] = 0
    u, v, w = g["key"] // g["V"], g["key"] % g["V"], g["w"].long()
    while True:
        new = dist.scatter_reduce(0, v, (dist[u] + w).clamp(max=INT_MAX), "amin")
        if torch.equal(new, dist):
            return dist.to(torch.int32)
        dist = new


def _brandes64(g, cols):
    """Dependencies of the sources, a level at a time; cols: per column, the sources
    (one of each disjoint graph) whose searches share it."""
    V, k = g["V"], len(cols)
    one = torch.ones(g["adj"].numel(), dtype=torch.float64, device=DEV)
    fwd = torch.sparse_csr_tensor(g["off"], g["adj"], one, (V, V))
    rev = fwd if g["roff"] is g["off"] else torch.sparse_csr_tensor(g["roff"], g["radj"], one, (V, V))
    sigma = torch.zeros((V, k), dtype=torch.float64, device=DEV)
    level = torch.full((V, k), -1, dtype=torch.int16, device=DEV)
    for j, s in enumerate(cols):
        s = torch.as_tensor(s, device=DEV).long()
        sigma[s, j] = 1.0
        level[s, j] = 0
    depth = 0
    while True:
        new = rev @ torch.where(level == depth, sigma, 0.0)
        at = (new > 0) & (level < 0)
        if not bool(at.any()):
            break
        depth += 1
        sigma = torch.where(at, new, sigma)
        level[at] = depth
    delta = torch.zeros_like(sigma)
    for d in range(depth - 1, 0, -1):
        q = torch.where(level == d + 1, (1.0 + delta) / sigma, 0.0)
        delta = torch.where(level == d, sigma * (fwd @ q), delta)
    return delta.sum(1)


def exact(case, seed):
    algo = case["algo"]
    if algo in ("tc", "clustering"):
        if case["n"] > 8192:  # whole numbers; the dense form is for small graphs
            return None
        count, per = _triangles64(_graph(case, seed))
        return count if algo == "tc" else per
    if algo == "louvain":  # the partition is the algorithm's own; its modularity goes with it
        return None
    if algo == "sssp":
        if case["graph"] == "grid":  # thousands of rounds
            return None
        g = _graph(case, seed)
        return _paths64(g, int(g["sources"][0]))
    g = _graph(case, seed)
    V = g["V"]
    if algo == "bc":
        src = g["sources"]
        return sum(_brandes64(g, [[v] for v in src[i:i + 32]]) for i in range(0, len(src), 32))
    if algo == "bc_graphs":
        src = g["sources"].reshape(case["graphs"], case["sources"])
        return sum(_brandes64(g, [src[:, j] for j in range(i, min(i + 8, case["sources"]))])
                   for i in range(0, case["sources"], 8))
    # Ranks: the iteration that ends the FP32 run depends on rounding, so the iteration
    # count and the last change have no 64-bit value of their own.
    one = torch.full((V,), 1.0 / V, dtype=torch.float64, device=DEV)
    if algo == "pagerank":
        return [_ranks64(g["off"], g["roff"], g["radj"], one, 100, 1e-6), None, None]
    gone, new = _batch(case, g)
    ranks = _ranks64(g["off"], g["roff"], g["radj"], one, 100, 1e-7).float().double()
    key = torch.unique(torch.cat([g["key"][~torch.isin(g["key"], gone)], new]))
    off, _ = _csr(V, key)
    roff, radj = _csr(V, torch.sort((key % V) * V + key // V).values)
    there = _ranks64(off, roff, radj, ranks, 100, 1e-6)
    back = _ranks64(g["off"], g["roff"], g["radj"], there, 100, 1e-6)
    return [[there, None, None], [back, None, None]]
