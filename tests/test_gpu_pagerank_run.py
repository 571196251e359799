"""GPU: PageRank's one launch for all iterations against the FP64 oracle at fixed iteration
counts, on both sides of the sizes from which one launch per iteration takes over: rows with
and without in-edges, rows split in chunks, one vertex, no edges, host and device output, and
a warm start.

Tolerance: L1 < 1e-6, the bound of the other PageRank tests (a rank is an FP64 sum rounded to
FP32 four times per iteration, errors decaying by the damping: 4 * 2^-24 / 0.15 = 1.6e-6 if
every rounding went the same way)."""
import numpy as np
import pytest

from graphs import empty, from_pairs, path, star
from oracle import oracle as O
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


def _hubs(n_edges):
    # 40 hubs of 2,040 to 2,079 in-edges (the chunk length is 2,048) and random rest
    rng = np.random.default_rng(n_edges)
    V = 60000
    hub = np.concatenate([np.full(2040 + h, h) for h in range(40)])
    dst = np.concatenate([hub, rng.integers(40, V // 2, n_edges - len(hub))])
    return from_pairs(V, np.stack([rng.integers(0, V, len(dst)), dst], 1))


GRAPHS = {
    "one": lambda: empty(1),
    "no_edges": lambda: empty(5000),
    "path": lambda: path(3),
    "star": lambda: star(5000),
    "rmat": lambda: G.rmat(12, 16, seed=2, directed=True),
    "hubs_below": lambda: _hubs(1_490_000),
    "hubs_above": lambda: _hubs(1_540_000),
    "er_below": lambda: G.erdos_renyi(180_000, 33, seed=5),
    "er_above": lambda: G.erdos_renyi(184_000, 33, seed=5),
}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_fixed_iterations_match_the_oracle(name):
    import torch

    g = GRAPHS[name]()
    g.ensure_reverse()
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        for iters in (1, 2, 3, 20):
            out, it, diff = dg.pagerank(0.0, 0.85, iters)
            ref, _, rdiff = O.pagerank(g.indexofNodes, g.rev_indexofNodes, g.srcList, 0.0, 0.85, iters,
                                       fixed_iters=iters)
            if it != iters:  # the FP32 ranks stopped changing: the oracle's change is at rounding level
                assert diff == 0.0 and rdiff < 1e-6
            assert np.abs(out.astype(np.float64) - ref).sum() < 1e-6, (name, iters)
            assert abs(diff - rdiff) < 1e-6
        dev = torch.empty(g.V, dtype=torch.float32, device="cuda")
        _, it2, diff2 = dg.pagerank(0.0, 0.85, 20, out=dev)
        assert (it2, diff2) == (it, diff) and np.array_equal(dev.cpu().numpy(), out)
        # a warm start from the ranks of 3 iterations continues the same run
        part, _, _ = dg.pagerank(0.0, 0.85, 3)
        none = (np.empty(0, "S1"), np.empty(0, np.int32), np.empty(0, np.int32), None)
        warm, _, _ = dg.pagerank_dynamic(*none, part, 0.0, 0.85, 17)
        assert np.abs(warm.astype(np.float64) - ref).sum() < 1e-6


@pytest.mark.parametrize("iters", [15, 16, 17, 24, 25, 60])
def test_first_call_stops_at_the_iteration_it_would(iters):
    # above the one-launch sizes a first call reads the stop test after 16, 24, 36 ...
    # iterations, a second launches them all: the same ranks, count and change
    g = GRAPHS["er_above"]() if iters == 60 else GRAPHS["hubs_above"]()
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        first = dg.pagerank(1e-6 if iters == 60 else 0.0, 0.85, iters)
        again = dg.pagerank(1e-6 if iters == 60 else 0.0, 0.85, iters)
        assert first[1] == again[1] and (iters == 60 or first[1] == iters)
        # the change is a sum over CTAs in one order, so it and the ranks are the same bits
        assert first[2] == again[2] and np.array_equal(first[0], again[0])


@pytest.mark.parametrize("order", [0, 1])
def test_transpose_of_rows_of_every_length(order):
    # rows of 0 to 4 entries, around a window (32), a warp's row (128) and a CTA's (1,024)
    rng = np.random.default_rng(3)
    degrees = np.concatenate([np.tile([0, 1, 2, 4, 31, 32, 33], 40), [127, 128, 129, 130, 1023, 1024, 1025, 3000]])
    V = 4000
    src = np.repeat(np.arange(len(degrees)), degrees)
    dst = np.concatenate([rng.choice(V, d, replace=False) for d in degrees])
    g = from_pairs(V, np.stack([src, dst], 1))
    g.ensure_reverse()
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        dg.tune_set("pr.order", order)
        out, _, _ = dg.pagerank(0.0, 0.85, 3)
    ref, _, _ = O.pagerank(g.indexofNodes, g.rev_indexofNodes, g.srcList, 0.0, 0.85, 3, fixed_iters=3)
    assert np.abs(out.astype(np.float64) - ref).sum() < 1e-6
