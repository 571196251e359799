"""GPU: sp_sssp_dynamic with a repair and additions from nearly every vertex in one batch. A
vertex that is both reset and the source of an added edge is queued once, so the queues'
V entries hold all seeds. Distances against the oracle, exact."""
import numpy as np
import pytest

from oracle import oracle as O
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,dels", [(20, 31, 12), (64, 64, 100), (101, 77, 300)])
def test_repair_with_additions_from_every_vertex(rows, cols, dels):
    g = G.grid(rows, cols)
    g.edgeLen = G.hash_weights(g, 3, 1, 50, True)
    source, V = (rows // 2) * cols + cols // 2, g.V
    rng = np.random.default_rng(7)
    u = np.repeat(np.arange(V, dtype=np.int32), np.diff(g.indexofNodes))
    held = set(zip(u.tolist(), g.edgeList.tolist()))
    with DeviceGraph.from_csr(g) as dg:
        dg.tune_set("sssp.repair", 1)
        dist, _ = dg.sssp(source)
        # tight edges into vertices far out: small subtrees, so that the repair runs
        tight = np.flatnonzero((dist[u] + g.edgeLen == dist[g.edgeList]) & (dist[g.edgeList] > np.quantile(dist, 0.7)))
        pick = rng.choice(tight, dels, replace=False)
        adds = [(a, b) for a, b in zip(range(V), rng.permutation(V).tolist()) if a != b and (a, b) not in held]
        s = np.concatenate([u[pick], [a for a, _ in adds]]).astype(np.int32)
        d = np.concatenate([g.edgeList[pick], [b for _, b in adds]]).astype(np.int32)
        w = np.concatenate([np.ones(dels), rng.integers(20, 400, len(adds))]).astype(np.int32)
        dg.sssp_dynamic("d" * dels + "a" * len(adds), s, d, w, source, dist)
        assert dg.tune_get("sssp.last_incremental") == 2
        assert dg.tune_get("sssp.last_marked") + len(adds) > V
    keep = np.ones(u.size, bool)
    keep[pick] = False
    src = np.concatenate([u[keep], s[dels:]])
    dst = np.concatenate([g.edgeList[keep], d[dels:]])
    wt = np.concatenate([g.edgeLen[keep], w[dels:]])
    order = np.lexsort((dst, src))
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=V))]).astype(np.int32)
    ref = O.sssp(off, dst[order].astype(np.int32), wt[order].astype(np.int32), source)
    assert np.array_equal(dist, ref)
