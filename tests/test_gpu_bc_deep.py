"""GPU: BC, levels and path counts on the graphs whose launch or pieces differ by their largest
degree: rows on both sides of the piece size (64), and grids and rings on both sides of the
degree (8) up to which fewer CTAs run. Against the oracle: 1e-5 relative, counts exact."""
import numpy as np
import pytest

from graphs import from_pairs, star
from oracle import oracle as O
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


def _ring(n, reach):  # every vertex joined to the next `reach`: degree 2 * reach
    i = np.repeat(np.arange(n, dtype=np.int32), reach)
    return from_pairs(n, np.stack([i, (i + np.tile(np.arange(1, reach + 1), n)) % n], 1), symmetrize=True)


def _ring9(n):  # degree 8, one vertex of degree 9
    i = np.repeat(np.arange(n, dtype=np.int32), 4)
    p = np.stack([i, (i + np.tile(np.arange(1, 5), n)) % n], 1)
    return from_pairs(n, np.concatenate([p, [[0, n // 2]]]), symmetrize=True)


GRAPHS = {
    "star64": lambda: star(64, directed_in=False),
    "star65": lambda: star(65, directed_in=False),
    "ring8": lambda: _ring(3001, 4),
    "ring9": lambda: _ring9(3001),
    "ring10": lambda: _ring(2000, 5),
    "grid": lambda: G.grid(61, 67),
}


@pytest.mark.parametrize("nsrc", [1, 16, 40, 64])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_degree_borders(name, nsrc):
    g = GRAPHS[name]()
    srcs = G.pick_sources(g, min(nsrc, g.V), seed=4, min_out_degree=0)
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        ref = O.bc(g.indexofNodes, g.edgeList, srcs)
        for _ in range(2):
            out = dg.bc(srcs).astype(np.float64)
            assert np.all(np.abs(out - ref) <= 1e-5 * np.abs(ref) + 1e-9 * max(1.0, ref.max()))
        lv, sg = dg.bfs_sigma(srcs)
        for k in (0, len(lv) - 1):
            rl, rs, _ = O.bfs_sigma(g.indexofNodes, g.edgeList, int(srcs[k]))
            assert np.array_equal(lv[k], rl)
            assert np.all(np.abs(sg[k] - rs) <= 1e-12 * rs)  # beyond 2^53 in the deep ones


@pytest.mark.parametrize("shape,counts", [((20, 20), [3, 0, 16, 1]), ((150, 4), [40, 33, 2, 70]), ((70, 75), [16, 5, 9, 1])])
def test_many_deep_graphs(shape, counts):
    # small grids and strips: a CTA per graph where that is expected to be faster, and one
    # union otherwise, against each graph by itself
    one = G.grid(*shape)
    n = one.V
    u = np.repeat(np.arange(n, dtype=np.int32), np.diff(one.indexofNodes))
    pairs = np.concatenate([np.stack([u, one.edgeList], 1) + n * k for k in range(4)])
    union = from_pairs(4 * n, pairs)
    srcs = [G.pick_sources(one, c, seed=k, min_out_degree=0) for k, c in enumerate(counts)]
    voff = (n * np.arange(5)).astype(np.int32)
    soff = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    ids = np.concatenate([s + n * k for k, s in enumerate(srcs)]).astype(np.int32)
    with DeviceGraph.from_csr(union, with_weights=False) as dg:
        out = dg.bc_graphs(voff, soff, ids).astype(np.float64)
    for k in range(4):
        ref = O.bc(one.indexofNodes, one.edgeList, srcs[k]) if counts[k] else np.zeros(n)
        assert np.all(np.abs(out[n * k:n * k + n] - ref) <= 1e-5 * np.abs(ref) + 1e-9 * max(1.0, ref.max())), k


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("nsrc", [1, 16, 64])
def test_levels_without_in_edges(directed, nsrc):
    # a call of few sources on a directed graph, and a first one on any graph without in-edges,
    # pushes; other calls (from 17 sources or 8 M entries times sources) gather: the same levels
    # and path counts
    g = G.rmat(15, 8, seed=5, directed=directed)
    assert (g.E * nsrc > 8_000_000) == (nsrc == 64)
    srcs = G.pick_sources(g, nsrc, seed=2, min_out_degree=0)
    with DeviceGraph(g.indexofNodes, g.edgeList, None, None, None) as dg:
        runs = [dg.bfs_sigma(srcs) for _ in range(3)]
        cc = [dg.closeness_unweighted(srcs) for _ in range(2)]
    with DeviceGraph(g.indexofNodes, g.edgeList, None, None, None) as dg:
        cc.append(dg.closeness_unweighted(srcs))
    for k in range(0, nsrc, 5):
        rl, rs, _ = O.bfs_sigma(g.indexofNodes, g.edgeList, int(srcs[k]))
        for lv, sg in runs:
            assert np.array_equal(lv[k], rl) and np.array_equal(sg[k], rs)
    assert np.array_equal(cc[0], cc[1]) and np.array_equal(cc[0], cc[2])
