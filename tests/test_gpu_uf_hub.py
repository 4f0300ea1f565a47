"""Union-find CC around its hub bitmap, against the CPU oracle.

The largest component is grown from the highest-degree vertex when its list
is long enough (one vertex in 256), by a second sweep when it is shorter
than one in 64: hub degrees on both sides of each bound, hubs whose id is
above or below the rest of their component, members reached only through
unsampled neighbours, and vertices of other components between them
(reference: src/cc/cc_kernels.cu:4-269).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("n,deg", [(257, 1), (1024, 3), (1024, 4), (1024, 5), (4096, 63), (4096, 64),
                                   (4096, 65), (100_000, 390), (100_000, 391), (100_000, 1600),
                                   (33, 32)])
@pytest.mark.parametrize("hub_last", [False, True])
def test_hub_bounds(T, O, n, deg, hub_last, budget):
    rng = np.random.default_rng(n + deg)
    hub = n - 1 if hub_last else 0
    leaves = rng.permutation(n - 1)[:deg] + (0 if hub_last else 1)
    # chains hang off the leaves and short cycles float free
    chain = rng.permutation(n)[: n // 3]
    free = rng.integers(0, n, n // 8)
    src = np.concatenate([np.full(deg, hub), chain[:-1], free])
    dst = np.concatenate([leaves, chain[1:], np.minimum(free + 1, n - 1)])
    c = O.from_edges(n, src.astype(np.uint32), dst.astype(np.uint32), symmetric=True)
    want = O.cc(c)
    with T.Graph.from_arrays(c.off, c.adj, "csr") as g:
        g.set_symmetric(True)
        g.plan(int(budget * g.ne * 4), block_bytes=4096)
        for _ in range(2):
            got, _ = g.run("cc", timeout_ms=20000)
            assert np.array_equal(got, want)
