"""Batched runs with host-resident edges and with few and many pending sources
per vertex, against the oracle's single runs.

Compaction reads a vertex's pending distances word by word up to 8 pending
sources and as a row above, and the bitmap words are handed out in one round
of the warps when SSSP has host-resident edges: groups of 1 to 64 sources from
one place (many pending at once) and from everywhere, vertex counts with one
word, a part of a round and a whole one (no counterpart in the reference).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("n", [30, 1025, 75_777, 151_553, 300_001])
@pytest.mark.parametrize("k", [1, 8, 9, 64])
def test_rows(T, O, n, k, budget):
    rng = np.random.default_rng(n + k)
    m = 5 * n
    c = O.from_edges(n, rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32))
    w = O.CSR(c.off, c.adj, rng.integers(1, 65, c.ne).astype(np.uint32))
    srcs = rng.integers(0, n, k)
    srcs[: k // 2] = c.adj[: k // 2] if k > 1 else srcs[:0]  # neighbours of one another's
    srcs = srcs.astype(np.uint32)
    check = sorted({0, 1, k // 2, k - 1} & set(range(k)))
    with T.Graph.from_arrays(w.off, w.wcsr_edges(), "wcsr") as g:
        g.plan(int(budget * g.ne * 4), block_bytes=1 << 16)
        got, sums, _ = g.batch_run("sssp", srcs, timeout_ms=20000)
        for i in check:
            assert np.array_equal(got[i], O.sssp(w, int(srcs[i])))
        for i in range(k):
            assert int(sums[i]) == T.values_checksum(got[i])
    with T.Graph.from_arrays(c.off, c.adj, "csr") as g:
        g.plan(int(budget * g.ne * 4), block_bytes=1 << 16)
        got, sums, _ = g.batch_run("bfs", srcs, timeout_ms=20000)
        for i in check:
            assert np.array_equal(got[i], O.bfs(c, int(srcs[i])))
