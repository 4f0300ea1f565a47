"""Batched runs where the split of the work over warps changes shape.

A warp takes 32 bitmap words (1,024 vertices) at a time on large graphs and
fewer on small ones, groups of small vertices shrink and chunks split into
parts while an iteration has few tasks: vertex counts around one word, one
word group and one warp's share, group sizes that leave a half-warp empty,
and a hub whose chunks split.  Every row must equal the single-source run of
the oracle (no counterpart in the reference).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1025, 5000, 75_777])
@pytest.mark.parametrize("k", [1, 5, 17, 64])
def test_rows_equal_single_runs(T, O, n, k):
    rng = np.random.default_rng(n + k)
    m = 6 * n
    src = np.concatenate([rng.integers(0, n, m), np.zeros(min(n, 3000))])
    dst = np.concatenate([rng.integers(0, n, m), np.arange(min(n, 3000))])
    c = O.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32))
    w = O.CSR(c.off, c.adj, rng.integers(1, 65, c.ne).astype(np.uint32))
    srcs = rng.integers(0, n, k).astype(np.uint32)
    check = range(0, k, 1 if k < 10 else 13)
    with T.Graph.from_arrays(w.off, w.wcsr_edges(), "wcsr") as g:
        got, _, _ = g.batch_run("sssp", srcs)
        for i in check:
            assert np.array_equal(got[i], O.sssp(w, int(srcs[i])))
    with T.Graph.from_arrays(c.off, c.adj, "csr") as g:
        got, _, _ = g.batch_run("bfs", srcs)
        for i in check:
            assert np.array_equal(got[i], O.bfs(c, int(srcs[i])))


@pytest.mark.parametrize("wmax", [1, 64, 65, 1 << 20, (1 << 32) - 1])
def test_default_window_follows_the_weights(T, O, wmax):
    c = O.rmat(12, 8)
    rng = np.random.default_rng(wmax % 1000)
    w = O.CSR(c.off, c.adj, rng.integers(1, wmax + 1, c.ne).astype(np.uint32))
    srcs = O.sources(c, 16).astype(np.uint32)
    with T.Graph.from_arrays(w.off, w.wcsr_edges(), "wcsr") as g:
        got, _, _ = g.batch_run("sssp", srcs)
    for i in range(0, 16, 5):
        assert np.array_equal(got[i], O.sssp(w, int(srcs[i])))
