"""What the engine is timed on: the work its users give it, through its public entry points.

A case names a task, a synthetic graph and how many sources or requests it has.  Graphs are
made on the GPU from a seed (RMAT with a=0.57 b=0.19 c=0.19, or Erdos-Renyi), without
self-loops and duplicate edges, weights uniform in [1, 63] and the same in both directions;
then they are taken through the library as host arrays, the way a program loads them.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "test-world_gb300"))
import ptgraph  # noqa: E402

SERVE_KINDS = (ptgraph.PTG_Q_BFS, ptgraph.PTG_Q_SSSP, ptgraph.PTG_Q_BFS, ptgraph.PTG_Q_PPR, ptgraph.PTG_Q_BFS,
               ptgraph.PTG_Q_SSSP, ptgraph.PTG_Q_BFS, ptgraph.PTG_Q_SSSP, ptgraph.PTG_Q_BFS, ptgraph.PTG_Q_PPR)
ITERS, DAMPING, WMAX = 20, 0.85, 63
FAR = 1 << 40  # unreached, in exact()


def listed():
    rmat = {"graph": "rmat", "edge_factor": 16, "symmetric": True, "shuffled": False, "wide": False}
    er = dict(rmat, graph="er", edge_factor=4)
    return [
        # one plain BFS on the small graph of the smallest configuration: launches and latency
        dict(rmat, name="bfs_rmat16", task="bfs", n=1 << 16, count=1),
        # the BFS part of the in-HBM suite: searches one after another on the benchmark's graph
        dict(rmat, name="bfs_rmat24", task="bfs", n=1 << 24, count=4),
        # the SSSP part of the suite: near/far buckets over 0.5 G weighted edges
        dict(rmat, name="sssp_rmat24", task="sssp", n=1 << 24, count=2),
        # components of a mid-sized graph whose ids carry no order, as ids of user data do
        dict(rmat, name="cc_ragged", task="cc", n=3000017, count=1, shuffled=True),
        # the PageRank part of the suite
        dict(rmat, name="pagerank_rmat24", task="pagerank", n=1 << 24, count=1),
        # personalized PageRank of a recommender's users: one full pass of 8 sources
        dict(rmat, name="ppr_batch_rmat20", task="ppr", n=1 << 20, count=8),
        # multi-source BFS of the batched configuration: one group of 256 sources
        dict(rmat, name="msbfs_rmat22", task="msbfs", n=1 << 22, count=256),
        # multi-source SSSP (distance tables for landmarks): two groups of 64 sources
        dict(rmat, name="mssssp_rmat20", task="mssssp", n=1 << 20, count=128),
        # components of a batch of uneven small graphs, handed over as host arrays
        dict(er, name="cc_batch_er", task="cc_batch", n=4000000, count=512),
        # a directed weighted graph of which half stays in pinned host memory and is streamed
        dict(rmat, name="ooc_sssp_rmat22", task="sssp_streamed", n=1 << 22, count=1, symmetric=False),
        # a burst of mixed requests on uploaded graphs of several sizes, through the server
        dict(rmat, name="serve_mix", task="serve", n=1 << 18, count=48),
        # a call of the drop-in API: host arrays with 8-byte edge records in, distances out
        dict(rmat, name="dropin_sssp", task="dropin_sssp", n=200003, count=1, symmetric=False),
    ]


def draw(rng):
    # task: smallest and largest n, largest count
    ranges = {"bfs": (1 << 10, 1 << 24, 4), "sssp": (1 << 10, 1 << 23, 2), "cc": (1 << 10, 1 << 23, 1),
              "pagerank": (1 << 10, 1 << 23, 1), "ppr": (1 << 10, 1 << 20, 8), "msbfs": (1 << 10, 1 << 21, 256),
              "mssssp": (1 << 10, 1 << 19, 128), "cc_batch": (1 << 14, 1 << 22, 512),
              "sssp_streamed": (1 << 20, 1 << 22, 1), "serve": (1 << 14, 1 << 18, 48),
              "dropin_sssp": (1 << 10, 1 << 18, 1), "dropin_bfs": (1 << 10, 1 << 19, 1),
              "dropin_cc": (1 << 10, 1 << 19, 1)}
    task = rng.choice(sorted(ranges))
    lo, hi, most = ranges[task]
    n = int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | rng.randint(0, 1)
    sym = task in ("pagerank", "ppr", "msbfs", "mssssp", "cc_batch", "serve") or rng.random() < 0.6
    if task.startswith("dropin") or task == "sssp_streamed":
        sym = False
    graph = "er" if task == "cc_batch" or rng.random() < 0.25 else "rmat"
    factor = rng.randint(8, 16)
    if graph == "er":  # components: sparse enough that there are several
        factor = rng.randint(1, 4) if task == "cc_batch" else rng.randint(1, 2) if task.endswith("cc") else rng.randint(3, 8)
    return {"task": task, "graph": graph, "n": n, "edge_factor": factor,
            "symmetric": sym, "shuffled": rng.random() < 0.5,
            "wide": not task.startswith("dropin") and task not in ("cc_batch", "serve") and rng.random() < 0.25,
            "count": int(math.exp(rng.uniform(0, math.log(most)))) if most > 1 else 1}


# ---------------------------------------------------------------------------
# graphs
# ---------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _mixed(x, seed):
    """A hash of int64 keys, well enough mixed for weights and even in both halves."""
    x = (x ^ (seed * 0x9E3779B9 + 0x7F4A7C15)) * 0x2545F4914F6CDD1D
    x = (x ^ ((x >> 29) & 0x7FFFFFFFF)) * 0x5851F42D4C957F2D
    return (x >> 33) & 0x3FFFFFFF


def _rmat_keys(n, m, gen):
    """Keys u * n + v of m RMAT draws over ids below n (draws outside are left out)."""
    keys = []
    scale = max(1, (n - 1).bit_length())
    for lo in range(0, m, 1 << 26):
        k = min(1 << 26, m - lo)
        u = torch.zeros(k, dtype=torch.int32, device="cuda")
        v = torch.zeros_like(u)
        for _ in range(scale):
            r = torch.rand(k, device="cuda", generator=gen)
            u += u + (r >= 0.76)
            v += v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        ok = (u < n) & (v < n) & (u != v)
        keys.append(u[ok].long() * n + v[ok])
    return torch.cat(keys)


def _er_keys(sizes, edge_factor, n, gen):
    """Keys of uniform draws inside each of several graphs that lie side by side."""
    m = sizes * edge_factor
    first = torch.repeat_interleave(torch.cumsum(sizes, 0) - sizes, m)
    size = torch.repeat_interleave(sizes, m)
    u, v = (first + torch.minimum((torch.rand(size.numel(), device="cuda", generator=gen, dtype=torch.float64)
                                   * size).long(), size - 1) for _ in range(2))
    return (u * n + v)[u != v]


def _edges(case, seed, n=None, sizes=None):
    """(offsets, targets, weights) on the GPU: int64, int64, int64."""
    n = n or case["n"]
    gen = _generator(seed)
    if case["graph"] == "rmat":
        key = _rmat_keys(n, n * case["edge_factor"], gen)
    else:
        sizes = torch.tensor([n], device="cuda") if sizes is None else sizes
        key = _er_keys(sizes, case["edge_factor"], n, gen)
    if case["shuffled"] and case["graph"] == "rmat":
        to = torch.randperm(n, device="cuda", generator=gen)
        key = to[key // n] * n + to[key % n]
    if case["symmetric"]:
        key = torch.cat([key, (key % n) * n + key // n])
    key = torch.unique(key)
    row, col = key // n, key % n
    del key
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    w = 1 + _mixed(torch.minimum(row, col) * n + torch.maximum(row, col), seed) % WMAX
    return off, col, w


def _host(x, dtype):
    """A pinned host array of the values (as a loader's read buffers are)."""
    y = torch.empty(x.numel(), dtype=dtype, pin_memory=True)
    y.copy_(x)
    return y.numpy().view(np.uint32 if dtype == torch.int32 else np.uint64)


def _sources(off, count, seed):
    """Vertices that have edges, drawn with the seed; ascending."""
    has = torch.nonzero(off[1:] > off[:-1]).flatten()
    at = (torch.rand(count, device="cuda", generator=_generator(seed + 7)) * has.numel()).long()
    return has[at.clamp(max=has.numel() - 1)].sort().values.cpu().numpy().astype(np.uint32)


def _batch_sizes(case, seed):
    """Vertices of each graph of a batch, log-uniform over a factor of 64, together n."""
    r = np.random.RandomState(seed % (1 << 31))
    x = np.exp(r.uniform(0, math.log(64), case["count"]))
    cut = np.round(np.cumsum(x) * case["n"] / x.sum()).astype(np.int64)
    return np.diff(cut, prepend=0)


def _serve_plan(case):
    """Sizes of the uploaded graphs, and (graph, kind) of each request: half BFS, a third SSSP, a fifth PPR."""
    sizes = [max(16, case["n"] >> s) + (s & 1) for s in (0, 1, 2, 3, 4, 6)]
    r = np.random.RandomState(case["n"] + case["count"])
    return sizes, [(int(r.randint(len(sizes))), SERVE_KINDS[i % len(SERVE_KINDS)]) for i in range(case["count"])]


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = ptgraph.Ctx(0)
    return _ctx


def _out(rows, n, dtype):
    return torch.empty((rows, n), dtype=dtype, device="cuda")


def prepare(case, seed):
    task, n, count = case["task"], case["n"], case["count"]
    s = {"task": task}
    if task == "cc_batch":
        sizes = _batch_sizes(case, seed)
        off, col, _ = _edges(case, seed, case["n"], torch.from_numpy(sizes).cuda())
        s["args"] = (np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64), off.cpu().numpy().astype(np.uint64),
                     col.cpu().numpy().astype(np.uint32))
        return s
    if task.startswith("dropin"):
        off, col, w = _edges(case, seed)
        edges = torch.stack([col, w], 1) if task == "dropin_sssp" else col
        s["name"] = {"dropin_sssp": "ssspCaculateInOpt", "dropin_bfs": "bfsCaculateInOpt", "dropin_cc": "ccCaculateInOpt"}[task]
        s["args"] = (off[:-1].cpu().numpy().astype(np.uint32), edges.cpu().numpy().astype(np.uint32))
        s["src"] = None if task == "dropin_cc" else int(_sources(off, 1, seed)[0])
        return s
    if task == "serve":
        sizes, plan = _serve_plan(case)
        server, gids, sources = ptgraph.Server(_context(), lanes=2), [], []
        for i, k in enumerate(sizes):
            off, col, w = _edges(case, seed + i, k)
            gids.append(server.upload(_host(off, torch.int64), _host(col, torch.int32), _host(w, torch.int32))[0])
            sources.append(_sources(off, len(plan), seed + i))
        s["server"] = server
        s["requests"] = [(gids[g], kind, int(sources[g][i]), np.zeros(sizes[g], np.float32 if kind == ptgraph.PTG_Q_PPR else np.uint32))
                         for i, (g, kind) in enumerate(plan)]
        return s
    off, col, w = _edges(case, seed)
    weighted = "sssp" in task
    config = None
    if task == "sssp_streamed":  # half of the edge bytes in HBM
        config = ptgraph.partition_config(device_budget_bytes=col.numel() * 4 + 2 * (32 << 20), force_out_of_core=1)
    s["graph"] = _context().graph(_host(off, torch.int64), _host(col, torch.int32), _host(w, torch.int32) if weighted else None,
                                  symmetric=case["symmetric"], config=config, pinned=True, wide_offsets=case["wide"])
    s["sources"] = _sources(off, count, seed)
    s["out"] = _out(count, n, torch.float32 if task in ("pagerank", "ppr") else torch.int32)
    return s


def run(state):
    task, dev = state["task"], ptgraph.PTG_OUT_DEVICE
    if task == "cc_batch":
        return _context().cc_batch(*state["args"])
    if task.startswith("dropin"):
        return ptgraph.compat.run(state["name"], *state["args"], state["src"])[1]
    if task == "serve":
        ids = [state["server"].submit(g, kind, src, out=out) for g, kind, src, out in state["requests"]]
        return [state["server"].wait(i)[0] for i in ids]
    g, out, sources = state["graph"], state["out"], state["sources"]
    if task == "bfs":
        for src, row in zip(sources, out):
            g.bfs(int(src), flags=dev, out=row)
    elif task in ("sssp", "sssp_streamed"):
        for src, row in zip(sources, out):
            g.sssp(int(src), flags=dev, out=row)
    elif task == "cc":
        g.cc(flags=dev, out=out[0])
    elif task == "pagerank":
        g.pagerank(iterations=ITERS, damping=DAMPING, flags=dev, out=out[0])
    elif task == "ppr":
        g.ppr_batch(sources, iterations=ITERS, damping=DAMPING, flags=dev, out=out)
    elif task == "msbfs":
        g.msbfs(sources, flags=dev, out=out)
    else:
        g.mssssp(sources, flags=dev, out=out)
    return out


def work(case):
    """The CSR read once and every result written once (edges counted as drawn: duplicates,
    a few per cent, are left out of the graph)."""
    def csr(n, weighted):
        m = n * case["edge_factor"] * (2 if case["symmetric"] else 1)
        return 4 * (n + 1) + m * (8 if weighted else 4), m

    if case["task"] == "serve":
        sizes, plan = _serve_plan(case)
        return {"bytes": sum(csr(k, True)[0] for k in sizes) + sum(4 * sizes[g] for g, _ in plan),
                "flops": sum(2 * ITERS * csr(sizes[g], True)[1] for g, kind in plan if kind == ptgraph.PTG_Q_PPR)}
    size, m = csr(case["n"], "sssp" in case["task"])
    rows = case["count"] if case["task"] not in ("cc", "cc_batch", "pagerank") else 1
    return {"bytes": size + 4 * case["n"] * rows,
            "flops": 2 * ITERS * m * rows if case["task"] in ("pagerank", "ppr") else 0}


# ---------------------------------------------------------------------------
# the results in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def _rows(off):
    return torch.repeat_interleave(torch.arange(off.numel() - 1, device="cuda"), off[1:] - off[:-1])


def _settle(x, row, col, w):
    """Fixed point of x[col] = min(x[col], x[row] + w)."""
    while True:
        y = x.scatter_reduce(0, col, x[row] + w, "amin")
        if torch.equal(x, y):
            return x
        x = y


def _from_source(off, row, col, w, src):
    x = torch.full((off.numel() - 1,), FAR, dtype=torch.int64, device="cuda")
    x[int(src)] = 1
    x = _settle(x, row, col, w)
    return torch.where(x >= FAR, torch.full_like(x, 0xFFFFFFFF), x)


def _ranks(off, row, col, src=None):
    """PageRank, or personalized PageRank of src (pull over a symmetric CSR)."""
    n = off.numel() - 1
    deg = (off[1:] - off[:-1]).double()
    start = torch.zeros(n, dtype=torch.float64, device="cuda")
    if src is None:
        start += 1.0 / n
    else:
        start[int(src)] = 1.0
    r = start
    for _ in range(ITERS):
        c = torch.where(deg > 0, r / deg.clamp(min=1), torch.zeros_like(r))
        dangling = r[deg == 0].sum()
        r = start * ((1 - DAMPING) + DAMPING * dangling) + DAMPING * torch.zeros_like(r).index_add_(0, row, c[col])
    return r


def _int32(x):
    """As the 32-bit output words read as signed numbers."""
    return torch.where(x > 0x7FFFFFFF, x - (1 << 32), x)


def exact(case, seed):
    task = case["task"]
    if task in ("msbfs", "mssssp", "sssp_streamed"):
        return None  # whole numbers, and many searches by full passes over the edges
    if task == "cc_batch":
        sizes = _batch_sizes(case, seed)
        off, col, _ = _edges(case, seed, case["n"], torch.from_numpy(sizes).cuda())
        row = _rows(off)
        first = torch.from_numpy(np.cumsum(sizes) - sizes).cuda().repeat_interleave(torch.from_numpy(sizes).cuda())
        x = _settle(torch.arange(off.numel() - 1, device="cuda"), row, col, 0)
        return x - first
    if task == "serve":
        sizes, plan = _serve_plan(case)
        found = [None] * len(plan)
        for i, k in enumerate(sizes):
            off, col, w = _edges(case, seed + i, k)
            row, sources = _rows(off), _sources(off, len(plan), seed + i)
            for j, (g, kind) in enumerate(plan):
                if g == i:
                    found[j] = (_ranks(off, row, col, sources[j]) if kind == ptgraph.PTG_Q_PPR else
                                _from_source(off, row, col, w if kind == ptgraph.PTG_Q_SSSP else 1, sources[j]))
        return found
    off, col, w = _edges(case, seed)
    row = _rows(off)
    if task in ("cc", "dropin_cc"):
        x = _settle(torch.arange(off.numel() - 1, device="cuda"), row, col, 0)
        return x if task == "dropin_cc" else x[None]
    if task == "pagerank":
        return _ranks(off, row, col)[None]
    sources = _sources(off, case["count"], seed)
    if task == "ppr":
        return torch.stack([_ranks(off, row, col, s) for s in sources])
    if task.startswith("dropin"):
        return _from_source(off, row, col, w if task == "dropin_sssp" else 1, sources[0])
    return torch.stack([_int32(_from_source(off, row, col, w if task == "sssp" else 1, s)) for s in sources])
