"""GPU: two host threads, each with its own graphs and a stream of its own, through the block cache
(more is released than it holds, so blocks are given up while the other thread allocates) and the
cooperative launches of PageRank, SSSP and BC; the results are those of one thread."""
import threading

import numpy as np
import pytest

from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


def _work(g, srcs, stream, rounds, big):
    import torch

    out = []
    for _ in range(rounds):
        with torch.cuda.stream(stream), DeviceGraph.from_csr(g) as dg:
            dg.set_stream(stream)
            pr = torch.empty(g.V, dtype=torch.float32, device="cuda")
            _, it, _ = dg.pagerank(1e-6, 0.85, 100, out=pr)
            r = [pr.cpu().numpy(), it, dg.tc(), dg.clustering_coeff(), dg.sssp(int(srcs[0]))[0]]
            if big:  # its rows, lists and scratch alone are above the cache's bound together
                r.append(dg.bc(srcs))
            out.append(r)
    return out


def test_two_threads():
    import torch

    small = G.rmat(13, 16, seed=3)
    large = G.rmat(21, 4, seed=4)
    for g in (small, large):
        g.edgeLen = G.hash_weights(g, 3, 1, 50, True)
        g.ensure_reverse()
    jobs = [(small, G.pick_sources(small, 20, seed=1), 12, True), (large, G.pick_sources(large, 64, seed=1), 2, True)]
    alone = [_work(g, s, torch.cuda.Stream(), 1, b)[0] for g, s, _, b in jobs]
    got = [None, None]

    def run(k):
        g, s, n, b = jobs[k]
        got[k] = _work(g, s, torch.cuda.Stream(), n, b)

    threads = [threading.Thread(target=run, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for ref, runs in zip(alone, got):
        assert runs is not None
        for r in runs:
            assert np.array_equal(r[0], ref[0]) and r[1:3] == ref[1:3]
            assert np.array_equal(r[3], ref[3]) and np.array_equal(r[4], ref[4])
            # dependencies of split entries are sums in any order
            assert np.all(np.abs(r[5].astype(np.float64) - ref[5]) <= 1e-6 * np.abs(ref[5]) + 1e-9)
