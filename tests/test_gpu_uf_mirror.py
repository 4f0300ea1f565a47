"""Union-find CC on graphs that are marked symmetric and are not.

thv_set_symmetric promises the labels of the weakly connected components
there.  In each graph below every edge is either among the first two of its
list or has its reverse, so that the sampled unions alone connect them: paths,
binary trees, and hubs whose neighbours lead on through one-way edges
(reference: src/cc/cc_kernels.cu:4-269).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def graph(name):
    if name.startswith("path"):
        n = int(name[4:])
        return n, np.arange(n - 1), np.arange(1, n)
    if name.startswith("tree"):
        n = int(name[4:])
        return n, (np.arange(1, n) - 1) // 2, np.arange(1, n)
    # hub 0 and its neighbours point at each other, chains lead away
    n, deg = 100_000, int(name[3:])
    leaves = np.arange(1, deg + 1)
    rest = np.arange(deg + 1, n)
    return n, np.r_[np.zeros(deg, int), leaves, rest - deg], np.r_[leaves, np.zeros(deg, int), rest]


@pytest.mark.parametrize("fmt", ["csr", "wcsr", "pairs"])
@pytest.mark.parametrize("budget", [0.0, 1.0])
@pytest.mark.parametrize("name", ["path5", "path200", "path600", "path20000", "tree300", "tree511",
                                  "hub380", "hub1500", "hub1600", "hub60000"])
def test_one_way_edges(T, O, name, budget, fmt):
    n, s, d = graph(name)
    c = O.from_edges(n, s.astype(np.uint32), d.astype(np.uint32))
    want = O.cc(O.from_edges(n, s.astype(np.uint32), d.astype(np.uint32), symmetric=True))
    w = np.random.default_rng(1).integers(1, 1 << 31, c.ne).astype(np.uint32)
    if fmt == "wcsr":
        w %= 64
    edges = c.adj if fmt == "csr" else np.stack([c.adj, w], 1)
    with T.Graph.from_arrays(c.off, edges, "csr" if fmt == "csr" else "wcsr") as g:
        assert g.mem_esz == (8 if fmt == "pairs" else 4)
        g.set_symmetric(True)
        assert g.symmetric
        g.plan(int(budget * g.ne * g.mem_esz), block_bytes=4096)
        got, _ = g.run("cc", timeout_ms=20000)
        assert np.array_equal(got, want)


def test_unbalanced_duplicates(T, O):
    """Reverses that occur less often than their edges: symmetric all the same."""
    s = O.rmat(12, 8, symmetric=True)
    first = s.adj[np.minimum(s.off[:-1], s.ne - 1).astype(np.int64)]
    deg = np.diff(s.off.astype(np.int64))
    keep = deg[:500] > 0
    off = s.off.astype(np.int64) + np.r_[0, np.cumsum(np.r_[keep, np.zeros(s.nv - 500, bool)])]
    adj = np.insert(s.adj, s.off[:500][keep].astype(np.int64), first[:500][keep])
    with T.Graph.from_arrays(off.astype(np.uint64), adj, "csr") as g:
        g.set_symmetric(True)
        g.plan()
        got, _ = g.run("cc", timeout_ms=20000)
        assert np.array_equal(got, O.cc(s))
