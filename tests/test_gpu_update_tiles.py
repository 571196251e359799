"""GPU: the merge of a batch of updates into the CSR equals the edge set after the batch, with
the batch's edges at and around the borders of the merge's tiles (4,096 entries): nothing but
deletions, nothing but additions, both on the same edge, repeats, and absent edges."""
import numpy as np
import pytest

from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu
TILE = 4096


def _case(name, g, src):
    E, V = g.E, g.V
    near = [i for t in range(0, E + 1, TILE) for i in (t - 1, t, t + 1) if 0 <= i < E]
    edge = [(int(src[i]), int(g.edgeList[i])) for i in near]
    have = set(zip(src.tolist(), g.edgeList.tolist()))
    new = [(s, (d + k) % V) for s, d in edge for k in (1, 2) if (s, (d + k) % V) not in have]
    if name == "deletions":
        return [("d", e) for e in edge]
    if name == "additions":
        return [("a", e) for e in dict.fromkeys(new)]
    if name == "held_again":
        return [("a", e) for e in edge] * 2
    if name == "both":
        return [("d", e) for e in edge[::2]] + [("a", e) for e in edge] + [("a", e) for e in new]
    if name == "absent":
        return [("d", e) for e in new] + [("d", edge[0])] * 3
    if name == "ends":
        return [("d", edge[0]), ("d", edge[-1]), ("a", (0, V - 1)), ("a", (V - 1, 0))]
    first = [("d", (int(s), int(d))) for s, d in zip(src[: 2 * TILE], g.edgeList[: 2 * TILE])]
    return first  # two whole tiles


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("name", ["deletions", "additions", "held_again", "both", "absent", "ends", "whole_tiles"])
def test_merge_at_tile_borders(name, weighted):
    g = G.rmat(11, 10, seed=4, directed=True)
    assert g.E > 3 * TILE
    src = np.repeat(np.arange(g.V), np.diff(g.indexofNodes)).astype(np.int32)
    g.edgeLen = G.hash_weights(g, 3, 1, 50, False)
    ups = _case(name, g, src)
    want = {(int(s), int(d)): int(w) for s, d, w in zip(src, g.edgeList, g.edgeLen)}
    for t, e in ups:
        if t == "d":
            want.pop(e, None)
    for i, (t, e) in enumerate(ups):
        if t == "a":
            want[e] = want.get(e, 0) + i % 5 + 1
    keys = sorted(want)
    with DeviceGraph.from_csr(g, with_weights=weighted) as dg:
        dg.update("".join(t for t, _ in ups), np.array([e[0] for _, e in ups], np.int32),
                  np.array([e[1] for _, e in ups], np.int32), np.array([i % 5 + 1 for i in range(len(ups))], np.int32))
        got = dg.export()
    off = np.searchsorted([k[0] for k in keys], np.arange(g.V + 1))
    assert np.array_equal(got["indexofNodes"], off)
    assert np.array_equal(got["edgeList"], [k[1] for k in keys])
    assert ("edgeLen" in got) == weighted
    if weighted:
        assert np.array_equal(got["edgeLen"], [want[k] for k in keys])
