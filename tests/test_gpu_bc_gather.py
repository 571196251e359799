"""GPU: BC in gather form where it can go wrong: batch sizes on both sides of each row width
(16, 32, 64 sources), split and whole entries, directed graphs (other rows for path counts
than for dependencies), and many graphs as one graph with uneven source counts, against
the oracle (1e-5 relative, path counts exact) and against the teams of CTAs."""
import numpy as np
import pytest

from graphs import clique, from_pairs, path, star
from oracle import oracle as O
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


def _close(out, ref):
    ref = np.asarray(ref, np.float64)
    bar = 1e-5 * np.abs(ref) + 1e-9 * max(1.0, float(np.abs(ref).max(initial=0.0)))
    return bool(np.all(np.abs(out.astype(np.float64) - ref) <= bar))


GRAPHS = {
    "rmat": lambda: G.rmat(10, 12, seed=2),
    "directed": lambda: G.rmat(11, 9, seed=6, directed=True),
    "star": lambda: star(777, directed_in=False),
    "star_in": lambda: star(700, directed_in=True),
    "clique": lambda: clique(67),
    "path": lambda: path(301),
    "grid": lambda: G.grid(17, 23),
}


@pytest.mark.parametrize("nsrc", [1, 16, 17, 32, 33, 64, 65])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_source_counts(name, nsrc):
    g = GRAPHS[name]()
    srcs = G.pick_sources(g, min(nsrc, g.V), seed=4, min_out_degree=0)
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        assert _close(dg.bc(srcs), O.bc(g.indexofNodes, g.edgeList, srcs))
        lv, sg = dg.bfs_sigma(srcs[:64])
        for k in (0, len(lv) - 1):
            rl, rs, _ = O.bfs_sigma(g.indexofNodes, g.edgeList, int(srcs[k]))
            assert np.array_equal(lv[k], rl) and np.array_equal(sg[k], rs)


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("counts", [[5, 0, 16, 1], [17, 33, 2, 70], [64, 64, 64, 64]])
def test_many_graphs_as_one(counts, directed):
    gs = [G.rmat(8, 6, seed=k, directed=directed) for k in range(3)] + [path(401)]
    voff = np.concatenate([[0], np.cumsum([g.V for g in gs])]).astype(np.int32)
    pairs, srcs, soff = [], [], [0]
    for k, g in enumerate(gs):
        u = np.repeat(np.arange(g.V, dtype=np.int32), np.diff(g.indexofNodes))
        pairs.append(np.stack([u, g.edgeList], 1) + voff[k])
        srcs.append(G.pick_sources(g, counts[k], seed=k, min_out_degree=0) + voff[k])
        soff.append(soff[-1] + len(srcs[-1]))
    union = from_pairs(int(voff[-1]), np.concatenate(pairs), name="union")
    s = np.concatenate(srcs).astype(np.int32)
    with DeviceGraph.from_csr(union, with_weights=False) as dg:
        out = dg.bc_graphs(voff, np.array(soff, np.int32), s)
        for k, g in enumerate(gs):
            ref = O.bc(g.indexofNodes, g.edgeList, srcs[k] - voff[k]) if counts[k] else np.zeros(g.V)
            assert _close(out[voff[k]:voff[k + 1]], ref), k
        dg.tune_set("bc.cluster", 1)  # a CTA per graph
        assert _close(dg.bc_graphs(voff, np.array(soff, np.int32), s), out)


def test_large_graph_with_wide_pieces():
    # above the size from which hubs are cut into fewer, longer pieces: dependencies as with
    # the small pieces (sums of the same terms, so to FP64 rounding before the FP32 store) and
    # as the oracle's
    g = G.rmat(19, 14, seed=6)
    assert g.E > 12_000_000 and np.diff(g.indexofNodes).max() > 2048
    srcs = G.pick_sources(g, 3, seed=1)
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        wide = dg.bc(srcs).astype(np.float64)
        dg.tune_set("bc.hub_deg", 64)
        dg.tune_set("bc.hub_chunk", 64)
        small = dg.bc(srcs).astype(np.float64)
    ref = O.bc(g.indexofNodes, g.edgeList, srcs)
    assert np.all(np.abs(wide - small) <= 2.0**-22 * np.abs(small))
    assert np.all(np.abs(wide - ref) <= 1e-5 * np.abs(ref) + 1e-6)
