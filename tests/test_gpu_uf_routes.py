"""Union-find CC on both sides of each line of its route, against the oracle.

A hub with `mids` neighbours, each with `leaves` more, and a ring of `ring`
vertices beside them: the ring sets the share of the edges that the hub's
neighbours own (1/16: below it there is no hub bitmap; 0.25 and 0.47: one
sweep or two), the leaves set its ratio to the hub's share of the vertices
(1.5).  The route is told by its launches: 6 without the bitmap, 7 with one
sweep, 8 with two (reference: src/cc/cc_kernels.cu:4-269).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# mids, leaves per mid (of all but the last two; of those), ring, launches
# resident, launches with host-resident edges
FORMS = {
    "below_reach": (64, 8, 8, 4033, 6, 6),
    "at_reach": (64, 8, 8, 4032, 8, 7),
    "below_link_two": (64, 8, 8, 577, 8, 7),
    "at_link_two": (64, 8, 8, 576, 8, 8),
    "below_one": (64, 8, 8, 37, 8, 8),
    "above_one": (64, 8, 8, 36, 7, 7),
    "above_share": (64, 2, 2, 0, 7, 7),
    "below_share": (64, 2, 1, 0, 6, 6),
    "wide": (20_000, 3, 3, 11, 7, 7),
}


def graph(O, name, seed):
    mids, leaves, last, ring, res, host = FORMS[name]
    per = np.full(mids, leaves)
    per[-2:] = last
    first = 1 + mids
    s = np.r_[np.zeros(mids, int), np.repeat(np.arange(1, first), per)]
    d = np.r_[np.arange(1, first), first + np.arange(per.sum())]
    n = first + int(per.sum())
    r = np.arange(ring)
    s, d, n = np.r_[s, n + r], np.r_[d, n + (r + 1) % max(ring, 1)], n + ring
    p = np.random.default_rng(seed).permutation(n)
    return O.from_edges(n, p[s].astype(np.uint32), p[d].astype(np.uint32), symmetric=True), res, host


@pytest.mark.parametrize("fmt", ["csr", "wcsr", "pairs"])
@pytest.mark.parametrize("budget", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("name", sorted(FORMS))
def test_route(T, O, name, budget, fmt):
    for seed in range(3):
        c, res, host = graph(O, name, seed)
        w = np.random.default_rng(1).integers(1, 64 if fmt == "wcsr" else 1 << 31, c.ne).astype(np.uint32)
        edges = c.adj if fmt == "csr" else np.stack([c.adj, w], 1)
        with T.Graph.from_arrays(c.off, edges, "csr" if fmt == "csr" else "wcsr") as g:
            assert g.mem_esz == (8 if fmt == "pairs" else 4)
            g.set_symmetric(True)
            g.plan(int(budget * g.ne * g.mem_esz), block_bytes=4096, small_list_degree=1)
            got, st = g.run("cc", timeout_ms=20000)
            assert st["kernel_launches"] == (res if budget == 1.0 else host)
            assert np.array_equal(got, O.cc(c))
