"""Push PageRank on resident graphs of more than three warp tiles per warp
(3.4 M edges or 909 K vertices on 148 SMs), which take a tile per CTA instead
of one per warp, against the FP64 oracle: 4-byte ids, packed weights and
pairs, with hubs above the 1,024 edges from which a row is split, empty rows
and vertices without out-edges (reference: src/pr/pr_kernels.cu :504-681,
:846-860).  Tolerance: contributions are rounded to FP32 once per
iteration (6e-8 relative) and contracted by 0.85, so 20 iterations stay below
4.1e-7 + 6e-8; 1e-6 is the engine's bound.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graphs(O):
    rng = np.random.default_rng(11)
    n = 400_003
    # flat rows around the CTA tile's 4,096 edges and 2,048 rows, and hubs
    # around its split bound and part size
    deg = np.where(np.arange(n) % 7 == 0, 0, 25)
    hubs = [1023, 1024, 1025, 4095, 4096, 4097, 8192, 12_289, 50_000]
    deg[rng.choice(n, len(hubs), replace=False)] = hubs
    deg[200_000:204_500] = 0
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.uint64)
    flat = O.CSR(off, rng.integers(0, n, int(off[-1])).astype(np.uint32))
    rmat = O.rmat(19, 24)
    return {k: (c, O.pagerank(c, 20)) for k, c in (("rows", flat), ("rmat", rmat))}


@pytest.mark.parametrize("fmt", ["csr", "wcsr", "pairs"])
@pytest.mark.parametrize("name", ["rows", "rmat"])
def test_resident_push(T, O, graphs, name, fmt):
    c, want = graphs[name]
    assert c.ne >= 8 << 20 and np.diff(c.off.astype(np.int64)).max() > 4096
    edges = c.adj if fmt == "csr" else np.stack([c.adj, (np.arange(c.ne) % 64 + 1).astype(np.uint32)], 1)
    with T.Graph.from_arrays(c.off, edges, "csr" if fmt == "csr" else "wcsr") as g:
        if fmt == "pairs":
            g.set_edge_packing(False)
        assert g.mem_esz == (8 if fmt == "pairs" else 4)
        assert g.plan(block_bytes=20_000_008)["host_edge_bytes"] == 0
        for _ in range(2):
            got, _ = g.run("pr_push", pr_iters=20)
            assert float(np.max(np.abs(got - want) / want)) <= 1e-6


@pytest.mark.parametrize("n,m", [(909_311, 400_000), (909_600, 400_000), (70_001, 3_409_800), (70_001, 3_410_500)])
def test_around_the_line(T, O, n, m):
    """Vertices or edges just below and above the line, mostly empty rows."""
    rng = np.random.default_rng(n + m)
    src = np.sort(rng.integers(0, n, m) // 3 * 3 % n)
    off = np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.uint64)
    c = O.CSR(off, rng.integers(0, n, m).astype(np.uint32))
    want = O.pagerank(c, 20)
    with T.Graph.from_arrays(c.off, c.adj, "csr") as g:
        assert g.plan()["host_edge_bytes"] == 0
        got, _ = g.run("pr_push", pr_iters=20)
    assert float(np.max(np.abs(got - want) / want)) <= 1e-6
