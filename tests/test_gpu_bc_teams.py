"""GPU: many graphs, a team of CTAs each, with level lists that fill in some teams while others
are at work. A path's vertex is listed once per source (its distances all differ), so 40
sources overflow the lists and the call runs again with 16 at a time; the other graphs'
teams must neither leave early nor stay behind. Against the oracle, 1e-5 relative."""
import numpy as np
import pytest

from graphs import from_pairs, path
from oracle import oracle as O
from starplat_b200 import _lib
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


def _union(gs, counts):
    voff = np.concatenate([[0], np.cumsum([g.V for g in gs])]).astype(np.int32)
    pairs, srcs = [], []
    for k, g in enumerate(gs):
        u = np.repeat(np.arange(g.V, dtype=np.int32), np.diff(g.indexofNodes))
        pairs.append(np.stack([u, g.edgeList], 1) + voff[k])
        srcs.append(G.pick_sources(g, counts[k], seed=k, min_out_degree=0))
    soff = np.concatenate([[0], np.cumsum([len(s) for s in srcs])]).astype(np.int32)
    ids = np.concatenate([s + b for s, b in zip(srcs, voff)]).astype(np.int32)
    return from_pairs(int(voff[-1]), np.concatenate(pairs), name="union"), voff, soff, ids, srcs


@pytest.mark.parametrize("cluster", [0, 1, 2, 4, 8])
def test_full_lists_in_some_teams(cluster):
    gs = [path(1501)] + G.er_batch(30, 100, 1200, 4, 12, seed=8) + [path(1301), path(1502)]
    counts = [40] + [40] * 30 + [40, 64]
    union, voff, soff, ids, srcs = _union(gs, counts)
    with DeviceGraph.from_csr(union, with_weights=False) as dg:
        if cluster:
            dg.tune_set("bc.cluster", cluster)
        for _ in range(2):  # the second call starts from what the first left
            out = dg.bc_graphs(voff, soff, ids).astype(np.float64)
            for k, g in enumerate(gs):
                ref = O.bc(g.indexofNodes, g.edgeList, srcs[k])
                got = out[voff[k]:voff[k + 1]]
                assert np.all(np.abs(got - ref) <= 1e-5 * np.abs(ref) + 1e-9 * max(1.0, ref.max())), k


@pytest.mark.parametrize("cluster", [1, 2, 8])
def test_too_deep_in_some_teams(cluster):
    # more levels than the form holds: refused, whatever the other teams do, and the handle
    # stays usable
    gs = [path(4300)] + G.er_batch(12, 100, 900, 4, 12, seed=2) + [path(4301)]
    union, voff, soff, ids, srcs = _union(gs, [3] * 14)
    ids = ids.copy()
    ids[[0, soff[13]]] = [0, voff[13]]  # an end of each path
    with DeviceGraph.from_csr(union, with_weights=False) as dg:
        dg.tune_set("bc.cluster", cluster)
        with pytest.raises(_lib.SPError):
            dg.bc_graphs(voff, soff, ids)
        assert dg.bc(ids[soff[2]:soff[3]]).max() > 0
