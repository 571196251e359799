"""GPU: Louvain's local move for whole weights (level 0) makes the plain form's moves: rows of
every length around one and two neighbours per lane, unit, whole and zero weights, and
weights that are not whole, which keep the general kernel."""
import numpy as np
import pytest

from graphs import clique, from_pairs, star
from oracle import oracle as O
from starplat_b200 import _lib
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


def _rings():
    # cliques of 28 .. 70 vertices, chained: degrees 27 .. 71 on both sides of 32 and 64
    pairs, base = [], 0
    for k in range(28, 71, 3):
        i, j = np.triu_indices(k, 1)
        pairs.append(np.stack([i, j], 1) + base)
        pairs.append(np.array([[base + k - 1, base + k]]))
        base += k
    return from_pairs(base + 1, np.concatenate(pairs), symmetrize=True, name="rings")


GRAPHS = {
    "sbm": lambda: G.sbm(6000, 20, exponent=2.0, avg_degree=34, p_in=0.7, seed=3),
    "rmat": lambda: G.rmat(12, 20, seed=5),
    "er": lambda: G.erdos_renyi(3000, 40, seed=2),
    "rings": _rings,
    "clique": lambda: clique(65),
    "star": lambda: star(70, directed_in=False),
    "directed": lambda: G.rmat(10, 12, seed=4, directed=True),
}


@pytest.mark.parametrize("weights", ["none", "ones", "whole", "zeros", "halves"])
@pytest.mark.parametrize("name", list(GRAPHS))
def test_same_moves_as_the_plain_form(name, weights):
    g = GRAPHS[name]()
    if weights == "none":
        w = None
    else:
        w = G.hash_weights(g, 7, 0 if weights == "zeros" else 1, 1 if weights == "ones" else 9, True)
        w = w.astype(np.float32) * (0.5 if weights == "halves" else 1.0)
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        q, comm, levels = dg.louvain(w)
        qp, commp, levelsp = dg.louvain(w, variant=_lib.SP_LV_PLAIN)
    assert levels == levelsp and np.array_equal(comm, commp) and abs(q - qp) < 1e-12
    assert abs(q - O.modularity(g.indexofNodes, g.edgeList, comm, w)) < 1e-9
