"""GPU: symmetry of graphs given without in-edges, found by looking for every entry's opposite:
one entry too few or too many at the places where blocks and their steps of 256 entries meet,
self-loops, and the in-edges that are made afterwards."""
import numpy as np
import pytest

from graphs import clique, empty, from_pairs, path, star
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


def _symmetric(off, adj):
    with DeviceGraph(off, adj, None, None, None) as dg:
        return dg.info()[2]


def _loops():
    i = np.arange(300, dtype=np.int32)
    return from_pairs(300, np.concatenate([np.stack([i, i], 1), np.stack([i[:-1], i[1:]], 1), np.stack([i[1:], i[:-1]], 1)]))


GRAPHS = {
    "empty": lambda: empty(5), "edge": lambda: path(2), "path": lambda: path(129), "star": lambda: star(2500, directed_in=False),
    "clique": lambda: clique(47), "rmat": lambda: G.rmat(12, 9, seed=2), "loops": _loops,
}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_symmetry_without_in_edges(name):
    g = GRAPHS[name]()
    assert _symmetric(g.indexofNodes, g.edgeList)
    with DeviceGraph(g.indexofNodes, g.edgeList, None, None, None) as dg:
        dg.info()
        x = dg.export()  # the in-edges of a symmetric graph are its out-edges
        assert np.array_equal(x["rev_indexofNodes"], g.indexofNodes) and np.array_equal(x["srcList"], g.edgeList)
    u = np.repeat(np.arange(g.V, dtype=np.int32), np.diff(g.indexofNodes))
    other = np.flatnonzero(u != g.edgeList)
    for e in {i for i in (0, 255, 256, 1023, 1024, g.E // 2, g.E - 1) if i in set(other.tolist())}:
        keep = np.delete(np.arange(g.E), e)
        h = from_pairs(g.V, np.stack([u[keep], g.edgeList[keep]], 1))
        assert not _symmetric(h.indexofNodes, h.edgeList), e


def test_directed_graphs():
    for g in (G.rmat(11, 8, seed=3, directed=True), star(700, directed_in=True), from_pairs(3, [[0, 1]])):
        with DeviceGraph(g.indexofNodes, g.edgeList, None, None, None) as dg:
            assert not dg.info()[2]
            x = dg.export()
            g.ensure_reverse()
            assert np.array_equal(x["rev_indexofNodes"], g.rev_indexofNodes) and np.array_equal(x["srcList"], g.srcList)
