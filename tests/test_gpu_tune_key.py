"""What a tuned batch configuration is kept by: the graph's shape, the SSSP
window that its weights lead to, and the kernel's way of splitting work (the
key's number), so that neither a graph with other weights nor a cache file of
the former kernel hands over its configuration.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_weights_and_kernel_are_part_of_the_key(T, O, tmp_path, monkeypatch):
    import torch

    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("THV_TUNE_CACHE", str(cache))
    c = O.rmat(11, 6, seed=77)
    srcs = O.sources(c, 64).astype(np.uint32)
    rng = np.random.default_rng(3)

    def graph(wmax):
        w = rng.integers(1, wmax + 1, c.ne).astype(np.uint32)
        return T.Graph.from_arrays(c.off, np.stack([c.adj, w], 1), "wcsr")

    with graph(255) as a, graph(100_000) as b:
        a.plan(), b.plan()
        assert a.mem_esz == b.mem_esz and a.ne == b.ne
        # a line of the key before the work split (version 3)
        p = b.plan_info()
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        cache.write_text("sssp3 nv=%d ne=%d esz=%d resident=%d blocks=%d sms=%d|16 256 512 16 32 4\n"
                         % (b.nv, b.ne, b.mem_esz, p["resident_edge_bytes"], p["num_blocks"], sms))
        assert b.batch_tuned("sssp")["tuned"] == 0
        a.batch_run("sssp", srcs, want_values=False, tune=True)
        assert a.batch_tuned("sssp")["tuned"] == 1
        assert b.batch_tuned("sssp")["tuned"] == 0
        assert a.batch_tuned("bfs")["tuned"] == 0
