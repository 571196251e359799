"""GPU: calls whose fastest form does not fit the free device memory run in a form that does.
Each test leaves a given number of bytes free (the rest is held by one allocation) and
compares with the same call made with all memory."""
import contextlib

import numpy as np
import pytest

from starplat_b200 import _lib
from starplat_b200 import generators as G
from starplat_b200.device import DeviceGraph

pytestmark = pytest.mark.gpu
MB = 1 << 20


@contextlib.contextmanager
def _only(free_bytes):
    """All but free_bytes of the device's free memory held for the block's time."""
    import torch

    _lib.lib().sp_cache_trim(None)
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - free_bytes, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def test_many_graphs_when_their_union_does_not_fit():
    # 300 random graphs of 8,000 vertices, 40 sources each: the union's rows, scratch, masks
    # and lists take 3.0 GB, a team per graph 1.8 GB; what the union had taken before it
    # failed must not be in the teams' way
    n, ng, k = 8000, 300, 40
    rng = np.random.default_rng(3)
    m = 2 * n
    u = rng.integers(0, n, (ng, m), dtype=np.int64) + n * np.arange(ng)[:, None]
    v = rng.integers(0, n, (ng, m), dtype=np.int64) + n * np.arange(ng)[:, None]
    u, v = u.ravel()[(u != v).ravel()], v.ravel()[(u != v).ravel()]
    V = n * ng
    key = np.unique(np.concatenate([u * V + v, v * V + u]))
    off = np.searchsorted(key, np.arange(V + 1) * V).astype(np.int32)
    adj = (key % V).astype(np.int32)
    voff = (n * np.arange(ng + 1)).astype(np.int32)
    soff = (k * np.arange(ng + 1)).astype(np.int32)
    srcs = np.concatenate([np.sort(rng.choice(n, k, replace=False)) + b for b in voff[:-1]]).astype(np.int32)
    with DeviceGraph(off, adj, None, off, adj) as dg:
        ref = dg.bc_graphs(voff, soff, srcs).astype(np.float64)
    with DeviceGraph(off, adj, None, off, adj) as dg:
        with _only(2850 * MB):
            out = dg.bc_graphs(voff, soff, srcs).astype(np.float64)
    assert np.all(np.abs(out - ref) <= 1e-5 * np.abs(ref) + 1e-6)


def test_batched_sssp_with_less_memory_than_a_full_batch():
    # a batch of 8 sources takes 8 * 37 bytes a vertex (1.2 GB here), 4 half of that
    g = G.grid(2048, 2048)
    g.edgeLen = G.hash_weights(g, 3, 1, 50, True)
    srcs = np.array([5, 77777, 2049, 4000000, 12345, 2000000, 3, 1048576], np.int32)
    with DeviceGraph.from_csr(g) as dg:
        dg.sssp(0)  # what a single solve keeps
        with _only(900 * MB):
            out = dg.sssp_batch(srcs)
        assert dg.tune_get("sssp.last_batch") == 4
        assert np.array_equal(out, dg.sssp_batch(srcs))
        assert dg.tune_get("sssp.last_batch") == 8


def test_triangles_when_the_rank_plan_does_not_fit():
    # making the lists in rank order takes about 26 bytes an entry (800 MB), the oriented
    # lists of the other kernels 10
    g = G.rmat(20, 16, seed=4)
    with DeviceGraph.from_csr(g, with_weights=False) as dg:
        count, per = dg.tc(), dg.clustering_coeff()
    for call, ref in (("tc", count), ("clustering_coeff", per)):
        with DeviceGraph.from_csr(g, with_weights=False) as dg:
            dg.info()  # the symmetry
            with _only(550 * MB):
                assert np.array_equal(getattr(dg, call)(), ref), call
            assert np.array_equal(getattr(dg, call)(), ref), call


@pytest.mark.parametrize("in_edges", [False, True])
def test_bc_when_in_edges_or_pieces_do_not_fit(in_edges):
    # 20 M directed edges on 50,000 vertices: in-edges take 0.4 GB to make and the gather form's
    # pieces 0.16 GB, where the push form takes 0.1 GB in all
    import torch

    V = 50000
    gen = torch.Generator(device="cuda").manual_seed(4)
    key = torch.unique(torch.randint(V * V, (20_200_000,), generator=gen, device="cuda"))
    key = key[key // V != key % V]
    off = torch.searchsorted(key, torch.arange(V + 1, device="cuda") * V).to(torch.int32)
    adj = (key % V).to(torch.int32)
    back = torch.sort(key % V * V + key // V).values
    roff = torch.searchsorted(back, torch.arange(V + 1, device="cuda") * V).to(torch.int32)
    rev = (roff, (back % V).to(torch.int32)) if in_edges else (None, None)
    del key, back
    srcs = np.arange(0, V, 800, dtype=np.int32)
    with DeviceGraph(off, adj, None, *rev) as dg:
        ref = dg.bc(srcs).astype(np.float64)
        lv, sg = dg.bfs_sigma(srcs[:20])
    with DeviceGraph(off, adj, None, *rev) as dg:
        with _only((150 if in_edges else 250) * MB):
            out = dg.bc(srcs).astype(np.float64)
        assert np.all(np.abs(out - ref) <= 1e-5 * np.abs(ref) + 1e-6)
        with _only((150 if in_edges else 250) * MB):
            lv2, sg2 = dg.bfs_sigma(srcs[:20])
        assert np.array_equal(lv, lv2) and np.array_equal(sg, sg2)
        again = dg.bc(srcs).astype(np.float64)  # with the memory back
    assert np.all(np.abs(again - ref) <= 1e-6 * np.abs(ref) + 1e-9)


def test_first_levels_when_the_push_form_does_not_fit():
    # without in-edges a first call pushes, in rows of 235 MB here; the gather form takes 60
    g = G.grid(512, 512)
    with DeviceGraph(g.indexofNodes, g.edgeList, None, None, None) as dg:
        ref = dg.bfs_sigma(np.array([70000], np.int32))
    with DeviceGraph(g.indexofNodes, g.edgeList, None, None, None) as dg:
        with _only(150 * MB):
            out = dg.bfs_sigma(np.array([70000], np.int32))
    assert np.array_equal(out[0], ref[0]) and np.all(np.abs(out[1] - ref[1]) <= 1e-12 * ref[1])
