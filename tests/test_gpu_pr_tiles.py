"""PageRank at the edges of its tiles, against the FP64 oracle.

A tile holds at most 480 edges and 128 rows, a lane sums 16 consecutive
edge slots, and rows of more than 480 edges are taken alone, in parts of
2,016: the degrees below put row ends on, before and after each of those
limits, with runs of empty rows and whole tiles without an edge (reference:
src/pr/pr_kernels.cu:23-160, :504-681).  Tolerance: contributions are rounded to FP32
once per iteration (6e-8 relative) and contracted by 0.85, so 20 iterations
stay below 4.1e-7 + 6e-8; 1e-6 is the engine's bound.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = {
    "spans": [15, 16, 17, 1, 0, 31, 32, 33, 0, 0, 2] * 300,
    "ones": [1] * 5000,
    "sparse": ([0] * 130 + [3] + [0] * 255 + [1, 0, 20]) * 3,
    "hubs": [479, 480, 481, 482, 511, 512, 513, 0, 2015, 2016, 2017, 5, 0, 4032, 4033, 1, 12277],
    "full_rows": [480] * 9 + [476, 4, 479, 1] + [120, 120, 120, 120] * 3,
    "no_edges": [0] * 2100,
}


@pytest.mark.parametrize("budget", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("name", sorted(DEGREES))
def test_pull_tile_edges(T, O, name, budget):
    deg = np.array(DEGREES[name], np.uint64)
    n = len(deg)
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    rng = np.random.default_rng(len(name))
    adj = rng.integers(0, n, int(off[-1])).astype(np.uint32)
    outdeg = np.bincount(adj, minlength=n).astype(np.uint32)
    want = O.pagerank_csc(off, adj, outdeg, 20)
    with T.Graph.from_arrays(off, adj, "csc", outdeg=outdeg) as g:
        # odd blocks: tiles start at every position inside a 16-byte word
        g.plan(int(budget * g.ne * 4), block_bytes=20_004)
        got, _ = g.run("pr_pull", pr_iters=20)
        again = g.values("pr_pull")
    assert float(np.max(np.abs(got - want) / want)) <= 1e-6
    assert np.array_equal(got, again)


@pytest.mark.parametrize("fmt", ["csr", "wcsr", "pairs"])
@pytest.mark.parametrize("budget", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("name", sorted(DEGREES))
def test_push_tile_edges(T, O, name, budget, fmt):
    deg = np.array(DEGREES[name], np.uint64)
    n = len(deg)
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    rng = np.random.default_rng(len(name) + 1)
    adj = rng.integers(0, n, int(off[-1])).astype(np.uint32)
    want = O.pagerank(O.CSR(off, adj), 20)
    edges = adj if fmt == "csr" else np.stack([adj, rng.integers(1, 65, len(adj)).astype(np.uint32)], 1)
    with T.Graph.from_arrays(off, edges, "csr" if fmt == "csr" else "wcsr") as g:
        if fmt == "pairs":
            g.set_edge_packing(False)
        g.plan(int(budget * g.ne * g.mem_esz), block_bytes=20_008, small_list_degree=1)
        got, _ = g.run("pr_push", pr_iters=20)
    assert float(np.max(np.abs(got - want) / want)) <= 1e-6
