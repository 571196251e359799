"""GPU: triangle counting in rank order (symmetric graphs) against the oracle, where its
kernel can go wrong: anchors with no, one and several work items, prefixes of every
length modulo the vector width, ranks on both sides of the exact bitmap's 16384, lists
that the hashed bitmap confuses, self-loops, and parts."""
import numpy as np
import pytest

from graphs import clique, empty, from_pairs, path, star
from oracle import oracle as O
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph
from starplat_b200.graph import CSRGraph

pytestmark = pytest.mark.gpu


def _loops():
    rng = np.random.default_rng(3)
    s, d = rng.integers(0, 300, (2, 4000)).astype(np.int32)
    loops = np.arange(0, 300, 3, dtype=np.int32)
    off, adj = G.csr_from_edges(300, np.concatenate([s, loops]), np.concatenate([d, loops]), symmetrize=True,
                                drop_self=False)
    return CSRGraph(off, adj, off, adj, name="loops")


def _hub_over_cold():
    # a hub joined to everything, over a ring with chords: most anchors have ranks above
    # 16384 and the hub's list of tasks spans many items
    n = 40000
    i = np.arange(1, n, dtype=np.int32)
    pairs = [np.stack([np.zeros_like(i), i], 1), np.stack([i[:-1], i[1:]], 1), np.stack([i[:-2], i[2:]], 1)]
    return from_pairs(n, np.concatenate(pairs), symmetrize=True, name="hub_over_cold")


CASES = {
    "empty": lambda: empty(5),
    "edge": lambda: path(2),
    "path": lambda: path(100),
    "star": lambda: star(3000, directed_in=False),
    "k3": lambda: clique(3),
    "k35": lambda: clique(35),
    "k300": lambda: clique(300),
    "loops": _loops,
    "rmat": lambda: G.rmat(13, 20, seed=3),
    "er_cold": lambda: G.erdos_renyi(40000, 60, seed=5),
    "hub_over_cold": _hub_over_cold,
    "rmat_cold": lambda: G.rmat(17, 12, seed=8),
}


@pytest.mark.parametrize("name", list(CASES))
def test_rank_order_counts(name):
    g = CASES[name]()
    ref, cf = O.tc(g.indexofNodes, g.edgeList), O.lcc(g.indexofNodes, g.edgeList)
    with DeviceGraph(g.indexofNodes, g.edgeList, None, g.rev_indexofNodes, g.srcList) as dg:
        assert dg.tc() == ref
        assert np.array_equal(dg.clustering_coeff(), cf)
        assert dg.tc() == ref  # the per-vertex pass leaves nothing behind
        assert sum(dg.tc_part(r, 3) for r in range(3)) == ref
        assert np.array_equal(sum(dg.clustering_coeff_part(r, 3) for r in range(3)), cf)
        dg.tune_set("tc.cta_warps", 2)
        dg.tune_set("tc.unroll", 1)
        assert dg.tc() == ref  # the bitmap or hash kernel
