"""GPU: the kernel knobs of TC and BC read back as what a call runs, writing that back changes
nothing, and a knob or variant that names a kernel runs it. Which kernel ran is told by the
launches of a repeated call: the count in rank order takes one, the hash kernel two (its
large anchors by themselves)."""
import numpy as np
import pytest

from oracle import oracle as O
from starplat_b200 import _lib
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu


def _launches(call):
    call()
    a = _lib.lib().sp_launch_count()
    r = call()
    return r, _lib.lib().sp_launch_count() - a


def test_tc_knobs_name_what_runs():
    g = G.rmat(17, 4, seed=3)  # above 65536 vertices
    ref = O.tc(g.indexofNodes, g.edgeList)
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        assert (dg.tune_get("tc.cta_warps"), dg.tune_get("tc.unroll")) == (-1, -1)
        assert _launches(dg.tc) == (ref, 1)
        for knob in ("tc.cta_warps", "tc.unroll"):
            dg.tune_set(knob, dg.tune_get(knob))
        assert _launches(dg.tc) == (ref, 1)
        dg.tune_set("tc.cta_warps", 4)  # names no kernel of graphs of this size
        assert _launches(dg.tc) == (ref, 1)
        for k in (1, 2, 4):
            dg.tune_set("tc.unroll", k)
            assert dg.tune_get("tc.unroll") == k
            assert _launches(dg.tc) == (ref, 2)
        dg.tune_set("tc.unroll", -1)
        assert _launches(dg.tc) == (ref, 1)
        dg.tune_set("tc.variant", 7)  # the hash kernel with four elements, its former default
        assert _launches(dg.tc) == (ref, 2)
        assert dg.tune_get("tc.last_variant") == 7
        dg.tune_set("tc.variant", -2)
        assert _launches(dg.tc) == (ref, 1)
        assert dg.tune_get("tc.last_variant") == -1
        for knob, bad in (("tc.cta_warps", -2), ("tc.cta_warps", 3), ("tc.unroll", 0), ("tc.unroll", -2)):
            with pytest.raises(_lib.SPError):
                dg.tune_set(knob, bad)


def test_bc_knobs_read_back_what_runs():
    small, large = G.rmat(10, 8, seed=2), G.rmat(19, 14, seed=6)
    assert large.E > 12_000_000
    for g, split in ((small, (64, 64)), (large, (256, 128))):
        with DeviceGraph.from_csr(g, with_weights=False) as dg:
            get = lambda: (dg.tune_get("bc.hub_deg"), dg.tune_get("bc.hub_chunk"))  # noqa: E731
            assert get() == split and dg.tune_get("bc.cluster") == 0
            dg.tune_set("bc.dir", 1)  # the push / pull form has one pair of defaults
            assert get() == (64, 64)
            dg.tune_set("bc.dir", 0)
            assert get() == split
            dg.tune_set("bc.hub_deg", 33)
            assert get() == (33, 64)
    with DeviceGraph.from_csr(small, with_weights=False) as dg:
        v = np.array([0, small.V], np.int32)
        s = G.pick_sources(small, 5, seed=1)
        a = dg.bc_graphs(v, np.array([0, 5], np.int32), s)
        dg.tune_set("bc.cluster", dg.tune_get("bc.cluster"))
        assert np.array_equal(a, dg.bc_graphs(v, np.array([0, 5], np.int32), s))


def test_bc_widest_and_narrowest_pieces_on_a_large_graph():
    # 70 M entries at the largest hub_deg and the smallest hub_chunk: the pieces' size is
    # raised until their number fits, without running over
    import torch

    V = 1 << 18
    gen = torch.Generator(device="cuda").manual_seed(4)
    a, b = torch.randint(V, (2, 38_000_000), generator=gen, device="cuda")
    key = torch.unique(torch.cat([a * V + b, b * V + a]))
    off = torch.searchsorted(key, torch.arange(V + 1, device="cuda") * V).to(torch.int32)
    adj = (key % V).to(torch.int32)
    assert adj.numel() > 1 << 26
    del a, b, key
    with DeviceGraph(off, adj, None, off, adj) as dg:
        ref = dg.bc(np.array([3], np.int32)).astype(np.float64)
        dg.tune_set("bc.hub_deg", 1 << 30)
        dg.tune_set("bc.hub_chunk", 1)
        out = dg.bc(np.array([3], np.int32)).astype(np.float64)
    assert np.all(np.abs(out - ref) <= 1e-6 * np.abs(ref))
