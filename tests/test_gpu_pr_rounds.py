"""PageRank over many rounds of warp tiles, against the FP64 oracle.

With host-resident edges tiles are handed out by place; resident graphs draw
them after the first round, several at a time from 152 K tiles.  A tile has at
most 128 rows, so many rows with few edges reach each of these, with the last
round full, nearly empty and in between (reference:
src/pr/pr_kernels.cu:23-160, :504-681).  Tolerance: contributions are rounded
to FP32 once per iteration (6e-8 relative) and contracted by 0.85, so the
result is off by less than 4.1e-7 + 6e-8; 1e-6 is the engine's bound.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sparse(O, n, m):
    rng = np.random.default_rng(n)
    src = np.sort(rng.integers(0, n, m) // 5 * 5 % n)
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.uint64)
    adj = rng.integers(0, n, m).astype(np.uint32)
    adj[::50] = rng.integers(0, 9, len(adj[::50]))
    return off, adj


@pytest.mark.parametrize("budget", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("n,m", [(600_001, 300_000), (610_007, 300_000), (1_300_000, 200_000),
                                 (4_300_001, 400_000), (4_900_003, 500_000)])
def test_rounds(T, O, n, m, budget):
    off, adj = sparse(O, n, m)
    od = np.bincount(adj, minlength=n).astype(np.uint32)
    want = O.pagerank_csc(off, adj, od, 6)
    with T.Graph.from_arrays(off, adj, "csc", outdeg=od) as g:
        g.plan(int(budget * g.ne * 4), block_bytes=100_004)
        got, _ = g.run("pr_pull", pr_iters=6)
    assert float(np.max(np.abs(got - want) / want)) <= 1e-6
    want = O.pagerank(O.CSR(off, adj), 6)
    with T.Graph.from_arrays(off, adj, "csr") as g:
        g.plan(int(budget * g.ne * 4), block_bytes=100_004, small_list_degree=1)
        got, _ = g.run("pr_push", pr_iters=6)
    assert float(np.max(np.abs(got - want) / want)) <= 1e-6


@pytest.mark.parametrize("budget", [0.0, 1.0])
def test_many_rounds(T, O, budget):
    n, m = 20_000_001, 600_000
    off, adj = sparse(O, n, m)
    od = np.bincount(adj, minlength=n).astype(np.uint32)
    want = O.pagerank_csc(off, adj, od, 3)
    with T.Graph.from_arrays(off, adj, "csc", outdeg=od) as g:
        g.plan(int(budget * g.ne * 4))
        got, _ = g.run("pr_pull", pr_iters=3)
    assert float(np.max(np.abs(got - want) / want)) <= 1e-6
    want = O.pagerank(O.CSR(off, adj), 3)
    with T.Graph.from_arrays(off, adj, "csr") as g:
        g.plan(int(budget * g.ne * 4), small_list_degree=1)
        got, _ = g.run("pr_push", pr_iters=3)
    assert float(np.max(np.abs(got - want) / want)) <= 1e-6
