"""GPU: the modularity that stops Louvain's first level, on rows of every length that its kernel
treats apart: up to and beyond 512 edges, and more long rows than a warp leaves to its CTA
(96, in its first four groups of 32 vertices). A threshold above every gain ends after the
first sweep, whose Q is that of the partition it returns; against the oracle, 1e-9."""
import numpy as np
import pytest

from graphs import from_pairs, star
from oracle import oracle as O
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


def _borders():  # hubs of 511, 512, 513, 767 .. 769 and 4097 leaves
    pairs, at = [], 7
    for h, n in enumerate((511, 512, 513, 767, 768, 769, 4097)):
        pairs.append(np.stack([np.full(n, h), np.arange(at, at + n)], 1))
        at += n
    return from_pairs(at, np.concatenate(pairs), symmetrize=True)


def _many_hubs():
    import torch

    warps = torch.cuda.get_device_properties(0).multi_processor_count * 6 * 8
    V = 32 * warps * 4 + 900
    hubs = np.concatenate([32 * warps * j + np.arange(32) for j in range(4)])  # one warp's
    rng = np.random.default_rng(5)
    ends = rng.integers(0, V, (hubs.size, 700))
    pairs = np.stack([np.repeat(hubs, 700), ends.ravel()], 1)
    return from_pairs(V, pairs[pairs[:, 0] != pairs[:, 1]], symmetrize=True)


GRAPHS = {"borders": _borders, "star": lambda: star(9000, directed_in=False), "rmat": lambda: G.rmat(14, 24, seed=4),
          "directed": lambda: G.rmat(13, 30, seed=4, directed=True), "many_hubs": _many_hubs}


@pytest.mark.parametrize("weights", ["none", "whole", "tenths"])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_first_level_modularity(name, weights):
    g = GRAPHS[name]()
    assert np.diff(g.indexofNodes).max() > 512
    w = None
    if weights != "none":
        w = G.hash_weights(g, 7, 1, 9, True).astype(np.float32) * np.float32(1.0 if weights == "whole" else 0.1)
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        q, comm, _ = dg.louvain(w, threshold=10.0)
        assert abs(O.modularity(g.indexofNodes, g.edgeList, comm, w) - q) < 1e-9
        q2, comm2, _ = dg.louvain(w, threshold=10.0)
    assert np.array_equal(comm, comm2) and q == q2  # the same on every run
