"""GPU: delta-stepping's row kernels are exact (distances equal the oracle's bit for bit) where
their paths change: rows of 0, 1 and 4 entries taken by one lane each and 5 and more flattened,
windows of 31 to 33 and 127 to 129 entries, rings that overflow in a cascade, hubs on both
sides of a piece and of a run of 8 pieces, with and without cascades and the dist filter."""
import numpy as np
import pytest

from graphs import empty, from_pairs, star
from oracle import oracle as O
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


def _rows(degrees, seed):
    # vertex i has degrees[i] out-edges to random vertices, some of them without out-edges
    rng = np.random.default_rng(seed)
    n = len(degrees)
    V = max(2 * n, 3 * max(degrees))
    src = np.concatenate([np.full(d, i) for i, d in enumerate(degrees)] + [np.arange(n - 1)])
    dst = np.concatenate([rng.choice(V, d, replace=False) for d in degrees] + [np.arange(1, n)])
    return from_pairs(V, np.stack([src, dst], 1))


GRAPHS = {
    "one": lambda: empty(1),
    "no_edges": lambda: empty(100),
    "up_to_4": lambda: _rows([0, 1, 4, 3, 2] * 300, 1),
    "up_to_5": lambda: _rows([4, 5, 0, 1] * 300, 2),
    "windows": lambda: _rows([31, 32, 33, 1, 0, 96, 127, 128] * 40, 3),
    "hubs": lambda: _rows([129, 63, 64, 65, 511, 512, 513, 2047, 2049, 5000] * 6, 4),
    "wide": lambda: _rows([100] * 2000, 5),
    "star": lambda: star(3000, directed_in=False),
    "grid": lambda: G.grid(70, 33),
}


@pytest.mark.parametrize("local", [0, 1, 64])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_distances_are_exact(name, local):
    g = GRAPHS[name]()
    w = G.hash_weights(g, 3, 0, 50, False)
    ref = {s: O.sssp(g.indexofNodes, g.edgeList, w, s) for s in {0, g.V // 2, g.V - 1}}
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        dg.tune_set("sssp.local", local)
        for filt in (-1, 0, 1):
            dg.tune_set("sssp.filter", filt)
            for delta in (7, 200, 10**6):
                for s, want in ref.items():
                    assert np.array_equal(dg.sssp(s, weight=w, delta=delta)[0], want), (filt, delta, s)
        rows = dg.sssp_batch(list(ref), weight=w)
        assert all(np.array_equal(np.asarray(r), want) for r, want in zip(rows, ref.values()))


def test_negative_weights_on_a_dag():
    rng = np.random.default_rng(6)
    a, b = np.sort(rng.integers(0, 3000, (2, 20000)), axis=0)
    g = from_pairs(3000, np.stack([a, b], 1)[a != b])
    w = rng.integers(-20, 60, g.E).astype(np.int32)
    want = O.sssp(g.indexofNodes, g.edgeList, w, 0)
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        for local in (0, 64):
            dg.tune_set("sssp.local", local)
            assert np.array_equal(dg.sssp(0, weight=w)[0], want)
