"""The traversals and rankings that a user of the engine runs, as timed cases.

Each case is one call of a public entry point on a graph that the program
already holds: BFS, SSSP, connected components, PageRank (pull and push),
batched multi-source BFS and SSSP, and BFS over a caller's own device arrays.
Graphs are RMAT (a=.57, b=.19, c=.19, permuted ids, duplicates and self-loops
removed: the engine's benchmark graphs) or uniform, made on the GPU from the
seed, with any vertex count.  The HBM edge budget is a fraction of the
format's edge bytes; what does not fit is read from pinned host memory.
Results land in pinned host buffers that the program keeps.

listed(), draw(rng), prepare(case, seed), run(state), work(case) and
exact(case, seed).
"""
import ctypes
import math

import numpy as np
import torch

import thievory_b200 as T

PR_ITERS = 20
DAMPING = 0.85
GROUP = 64  # sources of one batched group


def _case(algo, nv, ef, graph="rmat", budget=1.0, wmax=64, symmetric=False, name=None):
    """nv vertices, ef * nv edges drawn (symmetric: each inserted both ways);
    budget: HBM edge budget as a fraction of the format's edge bytes; wmax:
    weights are uniform in [1, wmax] (SSSP)."""
    c = {"algo": algo, "nv": nv, "ef": ef, "graph": graph, "budget": budget, "wmax": wmax,
         "symmetric": symmetric}
    return dict({"name": name}, **c) if name else c


def listed():
    return [
        # one query on a graph of a few thousand vertices: all of it is the
        # cost of starting, of the barriers between tiny levels, and of the
        # result's way back
        _case("bfs", 4999, 8, name="bfs-tiny"),
        # the latency path of a host framework that owns all device memory:
        # CSR and result stay in its own device arrays
        _case("bfs_noalloc", 150_001, 16, name="bfs-own-arrays"),
        # the benchmark's resident BFS (2^20 vertices, edge factor 16)
        _case("bfs", 1 << 20, 16, name="bfs-resident"),
        # BFS on a graph larger than its HBM budget: 60% of the edges over
        # the host link
        _case("bfs", 4_000_037, 16, budget=0.4, name="bfs-link"),
        # the benchmark's weighted workload at half its scale: weights in
        # [1, 64], stored packed, 40% of the WCSR bytes in HBM
        _case("sssp", 1 << 23, 16, budget=0.4, name="sssp-link"),
        # weights of a wide range (travel times, costs): {dst, w} pairs that
        # do not pack, flat degrees, all in HBM
        _case("sssp", 700_001, 6, graph="uniform", wmax=100_000, name="sssp-pairs"),
        # components of an undirected graph: sampling union-find
        _case("cc", 4_000_037, 8, budget=0.4, symmetric=True, name="cc-symmetric"),
        # components of a directed graph: min-label propagation, the
        # reference's method
        _case("cc", 1_000_003, 16, budget=0.4, name="cc-directed"),
        # PageRank, 20 iterations: pull over in-edges held in HBM, and push
        # over out-edges, half of them over the host link
        _case("pr_pull", 1 << 22, 16, name="pr-pull"),
        _case("pr_push", 3_000_017, 12, budget=0.5, name="pr-push"),
        # 64 queries in one traversal, every answer returned
        _case("batch_bfs", 1 << 18, 16, name="batch-bfs"),
        _case("batch_sssp", 150_001, 16, name="batch-sssp"),
    ]


# Largest vertex count x edge factor of a drawn case, by entry point (the
# listed sizes are the largest), and the smallest vertex count.
_MOST = {"bfs": 4_000_037 * 16, "sssp": (1 << 23) * 16, "cc": 4_000_037 * 8, "pr_pull": (1 << 22) * 16,
         "pr_push": 3_000_017 * 12, "batch_bfs": (1 << 18) * 16, "batch_sssp": 150_001 * 16,
         "bfs_noalloc": 1_500_000 * 16}


def draw(rng):
    algo = rng.choice(["bfs", "bfs", "bfs_noalloc", "sssp", "sssp", "cc", "pr_pull", "pr_push",
                       "batch_bfs", "batch_sssp"])
    ef = rng.randint(4, 24)
    most = _MOST[algo] // ef
    if algo == "pr_push":
        most = min(most, 3_000_017)
    nv = int(math.exp(rng.uniform(math.log(2000), math.log(most))))
    graph = rng.choice(["rmat", "rmat", "uniform"])
    budget = 1.0 if algo == "bfs_noalloc" else rng.choice([1.0, 1.0, 0.4, round(rng.uniform(0.1, 0.9), 3)])
    wmax = rng.choice([64, 64, 255, 100_000]) if "sssp" in algo else 64
    symmetric = algo == "cc" and rng.random() < 0.5
    if symmetric:
        ef = max(2, ef // 2)
    if algo == "pr_push" and budget < 1.0:
        budget = max(budget, 0.5)
    return _case(algo, nv, ef, graph, budget, wmax, symmetric)


# ------------------------------------------------------------------ inputs


def _edge_keys(case, gen, device):
    """Sorted keys src * nv + dst of the graph's distinct edges."""
    nv, raw = case["nv"], case["nv"] * case["ef"]
    if case["graph"] == "uniform":
        src = torch.randint(nv, (raw,), generator=gen, device=device)
        dst = torch.randint(nv, (raw,), generator=gen, device=device)
    else:
        a, b, c = 0.57, 0.19, 0.19
        scale = (nv - 1).bit_length()
        src = torch.zeros(raw, dtype=torch.int32, device=device)
        dst = torch.zeros(raw, dtype=torch.int32, device=device)
        for _ in range(scale):
            r = torch.rand(raw, generator=gen, device=device)
            down = r >= a + b
            right = ((r >= a) & ~down) | (r >= a + b + c)
            src.mul_(2).add_(down)
            dst.mul_(2).add_(right)
        perm = torch.randperm(nv, generator=gen, device=device)
        # 2^scale ids onto nv of them, keeping their order of popularity
        src = perm[(src.long() * nv) >> scale]
        dst = perm[(dst.long() * nv) >> scale]
    keep = src != dst
    src, dst = src[keep], dst[keep]
    if case["symmetric"]:
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    return torch.unique_consecutive(torch.sort(src * nv + dst).values)


def _graph(case, seed, device="cuda"):
    """(offsets, neighbour ids, weights or None, out-degrees) on the GPU; rows
    are sources, or destinations for pull PageRank (in-edges)."""
    gen = torch.Generator(device=device).manual_seed(int(seed))
    nv = case["nv"]
    keys = _edge_keys(case, gen, device)
    deg = torch.bincount(keys // nv, minlength=nv)
    if case["algo"] == "pr_pull":
        keys = torch.sort((keys % nv) * nv + keys // nv).values
        rows = torch.bincount(keys // nv, minlength=nv)
    else:
        rows = deg
    off = torch.zeros(nv + 1, dtype=torch.int64, device=device)
    torch.cumsum(rows, 0, out=off[1:])
    adj = (keys % nv).int()
    w = None
    if "sssp" in case["algo"]:
        w = torch.randint(1, case["wmax"] + 1, (adj.numel(),), generator=gen, device=device,
                          dtype=torch.int32)
    return off, adj, w, deg


def _sources(deg, seed, n):
    """n vertices uniform over those with out-edges."""
    gen = torch.Generator(device=deg.device).manual_seed(int(seed) + 1)
    have = torch.nonzero(deg).flatten()
    return have[torch.randint(have.numel(), (n,), generator=gen, device=deg.device)]


def prepare(case, seed):
    algo, nv = case["algo"], case["nv"]
    off, adj, w, deg = _graph(case, seed)
    # a single query starts at the best connected of eight vertices, so that
    # it reaches the graph's large component
    picks = _sources(deg, seed, GROUP)
    source = int(picks[:8][torch.argmax(deg[picks[:8]])])
    if algo == "bfs_noalloc":
        adj = torch.cat([adj, adj.new_zeros(64)])  # readable past its end
        return {"case": case, "off": off, "adj": adj, "ne": adj.numel() - 64, "source": source,
                "out": torch.empty(nv, dtype=torch.int32, device="cuda")}
    edges = adj if w is None else torch.stack([adj, w], dim=1)
    fmt = "wcsr" if w is not None else "csc" if algo == "pr_pull" else "csr"
    g = T.Graph.from_arrays(off.cpu().numpy().view(np.uint64), edges.cpu().numpy().view(np.uint32), fmt,
                            outdeg=deg.int().cpu().numpy().view(np.uint32) if fmt == "csc" else None)
    if case["symmetric"]:
        g.set_symmetric(True)
    pagerank = algo.startswith("pr")
    g.plan(None if case["budget"] >= 1.0 else int(case["budget"] * g.ne * g.esz),
           small_list_degree=1 if pagerank else 0)
    state = {"case": case, "graph": g, "source": source}
    if algo.startswith("batch"):
        state["sources"] = picks.int().cpu().numpy().view(np.uint32)
        state["out"] = torch.empty((GROUP, nv), dtype=torch.int32, pin_memory=True)
        state["sums"] = torch.empty(GROUP, dtype=torch.int64, pin_memory=True)
    else:
        state["out"] = torch.empty(nv, dtype=torch.float64 if pagerank else torch.int32, pin_memory=True)
        state["view"] = state["out"].numpy().view(np.float64 if pagerank else np.uint32)
    return state


# --------------------------------------------------------------------- run


def run(state):
    case = state["case"]
    algo = case["algo"]
    if algo == "bfs_noalloc":
        levels = ctypes.c_uint64()
        s = T.load_library().thv_bfs_noalloc(state["off"].data_ptr(), state["adj"].data_ptr(), case["nv"],
                                             state["ne"], state["source"], state["out"].data_ptr(), None,
                                             ctypes.byref(levels))
        assert s == T.THV_OK, T.load_library().thv_last_error()
        return state["out"]
    g = state["graph"]
    if algo.startswith("batch"):
        src = state["sources"]
        s = T.load_library().thv_batch_run(g._h, T.ALGO[algo[6:]], src.ctypes.data, len(src), None,
                                           state["out"].data_ptr(), state["sums"].data_ptr(), None)
        assert s == T.THV_OK, T.load_library().thv_last_error()
        return {"values": state["out"], "checksums": state["sums"]}
    if algo.startswith("pr"):
        g.run(algo, pr_iters=PR_ITERS, pr_damping=DAMPING, out=state["view"])
    else:
        g.run(algo, source=state["source"], out=state["view"])
    return state["out"]


def work(case):
    """The graph once (offsets, edges as given) and the result once; PageRank
    reads the edges in each of its iterations.  Duplicate edges, a few percent
    of an RMAT graph's, are counted here as if they were there."""
    nv, ne = case["nv"], case["nv"] * case["ef"] * (2 if case["symmetric"] else 1)
    algo = case["algo"]
    esz = 8 if "sssp" in algo else 4
    sweeps = PR_ITERS if algo.startswith("pr") else 1
    out = nv * (8 if algo.startswith("pr") else 4) * (GROUP if algo.startswith("batch") else 1)
    return {"bytes": nv * 8 + ne * esz * sweeps + out, "flops": 2 * ne * sweeps if algo.startswith("pr") else 0}


# ------------------------------------------------------------------- exact


def exact(case, seed):
    """PageRank in 64 bits: fixed iterations, dangling mass spread evenly.
    The other entry points return whole numbers."""
    if not case["algo"].startswith("pr"):
        return None
    off, adj, _, deg = _graph(case, seed)
    nv = case["nv"]
    rows = torch.repeat_interleave(torch.arange(nv, device="cuda"), off[1:] - off[:-1])
    src, dst = (adj.long(), rows) if case["algo"] == "pr_pull" else (rows, adj.long())
    r = torch.full((nv,), 1.0 / nv, dtype=torch.float64, device="cuda")
    d = deg.double()
    for _ in range(PR_ITERS):
        share = torch.where(deg > 0, r / d.clamp(min=1), 0.0)
        dangling = r[deg == 0].sum()
        r = (1 - DAMPING) / nv + DAMPING * (torch.zeros_like(r).index_add_(0, dst, share[src]) + dangling / nv)
    return r.cpu()
