"""GPU: PageRank with beta = 0, which asks for all iterations, on both sides of the size from which
they run as launches: the ranks, count and change of a call that may stop early and does not."""
import numpy as np
import pytest

from oracle import oracle as O
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [120_000, 126_000, 140_000])
@pytest.mark.parametrize("iters", [1, 17, 40])
def test_all_iterations(V, iters):
    g = G.erdos_renyi(V, 32, seed=V)
    assert abs(g.E - 4_000_000) < 600_000
    g.ensure_reverse()
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        runs = [dg.pagerank(b, 0.85, iters) for b in (0.0, 0.0, 0.0, 1e-30)]
    # the change can be exactly zero only after the ranks have stopped moving
    assert all(r[1] == runs[0][1] for r in runs) and (runs[0][1] == iters or runs[0][2] == 0.0)
    ref, _, rdiff = O.pagerank(g.indexofNodes, g.rev_indexofNodes, g.srcList, 0.0, 0.85, iters, fixed_iters=iters)
    for out, _, diff in runs:
        assert np.abs(out.astype(np.float64) - ref).sum() < 1e-6 and abs(diff - rdiff) < 1e-6
