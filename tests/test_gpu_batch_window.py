"""The default window of batched SSSP where distances span several windows.

The window is four times the largest weight or eight times the mean one,
within 256 .. 2^22.  Distances end at the vertex count, so the graphs have
vertices to spare; every row must equal the oracle's single-source run, and a
few long edges must not make the batch expand more than the window of the
other weights does (reference: src/sssp/sssp_kernels.cu, one source at a time).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def grid(O, rows, cols, nv=0):
    v = np.arange(rows * cols).reshape(rows, cols)
    s = np.r_[v[:, :-1].ravel(), v[:-1].ravel()].astype(np.uint32)
    d = np.r_[v[:, 1:].ravel(), v[1:].ravel()].astype(np.uint32)
    return O.from_edges(max(nv, rows * cols), s, d, symmetric=True)


# name: (rows, cols, vertices, largest weight, packed bytes per edge)
GRIDS = {"narrow": (150, 200, 0, 64, 4), "wide": (40, 60, 300_000, 5000, 4), "pairs": (40, 60, 300_000, 5000, 8),
         "past_cap": (2, 8, 9_000_000, 2_500_000, 8)}


@pytest.mark.parametrize("name", sorted(GRIDS))
def test_rows_over_many_windows(T, O, name):
    rows, cols, nv, wmax, esz = GRIDS[name]
    c = grid(O, rows, cols, nv)
    rng = np.random.default_rng(wmax)
    w = O.CSR(c.off, c.adj, rng.integers(1, wmax + 1, c.ne).astype(np.uint32))
    window = min(max(256, 4 * min(int(w.w.max()), -(-2 * int(w.w.sum(dtype=np.uint64)) // c.ne))), 1 << 22)
    srcs = rng.integers(0, rows * cols, 7).astype(np.uint32)
    with T.Graph.from_arrays(w.off, w.wcsr_edges(), "wcsr") as g:
        if esz == 8:
            g.set_edge_packing(False)
        assert g.mem_esz == esz
        got, _, _ = g.batch_run("sssp", srcs, timeout_ms=20000)
    for i, s in enumerate(srcs):
        want = O.sssp(w, int(s))
        reached = want[want <= c.nv]
        assert len(reached) > 4 and reached.max() > window
        assert np.array_equal(got[i], want)


@pytest.mark.parametrize("long_edges", [1, 100])
def test_few_long_edges_leave_the_window(T, O, long_edges):
    c = grid(O, 300, 200)
    rng = np.random.default_rng(long_edges)
    weights = rng.integers(1, 65, c.ne).astype(np.uint32)
    weights[rng.choice(c.ne, long_edges, replace=False)] = 10_000
    w = O.CSR(c.off, c.adj, weights)
    srcs = rng.integers(0, c.nv, 64).astype(np.uint32)
    with T.Graph.from_arrays(w.off, w.wcsr_edges(), "wcsr") as g:
        got, _, st = g.batch_run("sssp", srcs, timeout_ms=20000)
        fixed, _, st0 = g.batch_run("sssp", srcs, timeout_ms=20000, sssp_delta=256)
    assert np.array_equal(got, fixed)
    for i in (0, 31, 63):
        assert np.array_equal(got[i], O.sssp(w, int(srcs[i])))
    assert st["edges_expanded"] <= 1.25 * st0["edges_expanded"]
