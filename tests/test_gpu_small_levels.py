"""BFS levels inside one CTA: thv_bfs_noalloc on both sides of its edge bound,
and many short runs in a row, against the CPU oracle.

thv_bfs_noalloc runs levels of a few vertices in one CTA below 8 M edges and
every level on the grid above; its iteration count stops at the first level
without out-edges either way.  Small resident graphs hand levels back and
forth between one CTA and the grid every few microseconds, so each run must
leave alone what slower blocks still read (reference: src/bfs/bfs.cu:55-524).
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph(O, name):
    if name == "path":
        return O.from_edges(3000, np.arange(2999), np.arange(1, 3000)), 0
    if name == "isolated_source":
        return O.from_edges(100, np.arange(1, 99), np.arange(2, 100)), 0
    if name == "star":
        return O.from_edges(5000, np.zeros(4999, np.uint32), np.arange(1, 5000)), 0
    if name == "into_star":
        return O.from_edges(5001, np.r_[1, 2, np.full(4990, 3)], np.r_[2, 3, np.arange(10, 5000)]), 1
    g = O.rmat(*{"below": (19, 16), "above": (19, 18)}[name])
    assert (g.ne < 8 << 20) == (name == "below")
    return g, int(O.sources(g, 1)[0])


@pytest.mark.parametrize("name", ["path", "isolated_source", "star", "into_star", "below", "above"])
def test_noalloc(T, O, name):
    import torch

    g, src = graph(O, name)
    want = O.bfs(g, src)
    dev = torch.device("cuda:0")
    d_off = torch.from_numpy(g.off.view(np.int64)).to(dev)
    d_adj = torch.from_numpy(np.r_[g.adj, np.zeros(64, np.uint32)].view(np.int32)).to(dev)
    d_out = torch.empty(g.nv, dtype=torch.int32, device=dev)
    it = ctypes.c_uint64()
    lib = T.load_library()
    for _ in range(3):
        d_out.fill_(-1)
        torch.cuda.synchronize()
        st = lib.thv_bfs_noalloc(d_off.data_ptr(), d_adj.data_ptr(), g.nv, g.ne, src, d_out.data_ptr(),
                                 None, ctypes.byref(it))
        assert st == 0, lib.thv_last_error()
        assert np.array_equal(d_out.cpu().numpy().view(np.uint32), want)
        # level l holds value l + 1; the run ends at the first level whose
        # vertices have no out-edges
        deg = np.diff(g.off.astype(np.int64))
        out = np.bincount(want[want <= g.nv], weights=deg[want <= g.nv], minlength=g.nv + 3)
        assert it.value == int(np.flatnonzero(out[1:] == 0)[0])


@pytest.mark.parametrize("nv,ef", [(2000, 2), (2400, 8), (5000, 8), (20_000, 16)])
def test_many_short_runs(T, O, nv, ef):
    rng = np.random.default_rng(nv)
    c = O.from_edges(nv, rng.integers(0, nv, nv * ef).astype(np.uint32),
                     (rng.integers(0, nv, nv * ef) ** 2 // nv).astype(np.uint32))
    srcs = [int(s) for s in O.sources(c, 12)]
    want = {s: T.values_checksum(O.bfs(c, s)) for s in srcs}
    with T.Graph.from_arrays(c.off, c.adj, "csr") as g:
        g.plan()
        for _ in range(25):
            for s in srcs:
                _, st = g.run("bfs", source=s, want_values=False, checksum=True, timeout_ms=5000)
                assert st["checksum"] == want[s]
