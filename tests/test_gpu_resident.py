"""The one-launch traversal of in-HBM graphs at its edges: degrees around the
three work lists and a warp's pieces, one CTA and many, long chains (many
levels, many buckets), every offset width and vertex order, against the oracle."""
import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def csr(n, src, dst, symmetric, seed):
    if symmetric:
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    key = np.unique(src.astype(np.int64) * n + dst)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    row, col = key // n, key % n
    w = (1 + (np.minimum(row, col) * 7919 + np.maximum(row, col) * 31 + seed) % 63).astype(np.uint32)
    return off, col.astype(np.uint32), w


def hubs(degrees, seed):
    """Hubs of the given degrees over shared random leaves, and a chain through the hubs."""
    rng = np.random.RandomState(seed)
    n = len(degrees) + max(degrees) + 37
    ids = rng.permutation(n)
    src, dst = [], []
    for i, d in enumerate(degrees):
        src.append(np.full(d, ids[i]))
        dst.append(ids[len(degrees) + rng.permutation(n - len(degrees))[:d]])
        if i:
            src.append(ids[i - 1:i])
            dst.append(ids[i:i + 1])
    return n, np.concatenate(src), np.concatenate(dst), int(ids[0])


def chain(length, seed):
    ids = np.random.RandomState(seed).permutation(length)
    return length, ids[:-1], ids[1:], int(ids[0])


def random_graph(n, m, seed):
    rng = np.random.RandomState(seed)
    a, b = rng.randint(0, n, m), rng.randint(0, n, m)
    keep = a != b
    return n, a[keep], b[keep], int(a[0])


GRAPHS = {
    "edge_degrees": lambda: hubs([1, 15, 16, 17, 31, 64, 127, 128, 129, 255, 256, 257, 511, 513, 4097], 1),
    "chain": lambda: chain(700, 2),
    "one_cta": lambda: random_graph(60, 300, 3),
    "sparse": lambda: random_graph(5001, 9000, 4),
    "dense": lambda: random_graph(1999, 300000, 5),
    "large": lambda: random_graph(300007, 2500000, 6),
}


@pytest.mark.parametrize("name", GRAPHS)
@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("grouped", [False, True])
def test_traversals_match_oracle(ptg, ctx, ctx_grouped, oracle, name, symmetric, wide, grouped):
    n, src, dst, s = GRAPHS[name]()
    off, col, w = csr(n, src, dst, symmetric, n)
    G = (ctx_grouped if grouped else ctx).graph(off, col, w, symmetric=symmetric, wide_offsets=wide)
    ref = oracle.bfs(off, col, s, method="queue")
    st = {}
    assert (G.bfs(s, stats=st) == ref).all()
    assert st["iterations"] == ref[ref != 0xFFFFFFFF].max()  # one level per distance, the last finds nothing
    assert (G.bfs(s, flags=ptg.PTG_NO_DIRECTION_OPT) == ref).all()
    dist = oracle.sssp(off, col, w, s)
    for delta in (0, 1, 7, 1000000):
        assert (G.sssp(s, delta=delta) == dist).all(), delta
    assert (G.sssp(s, flags=ptg.PTG_REFERENCE_SCHEDULE | ptg.PTG_LEVEL_ZERO_BASED) ==
            np.where(dist == 0xFFFFFFFF, dist, dist - 1)).all()
    assert (G.cc(flags=ptg.PTG_REFERENCE_SCHEDULE) == oracle.cc(off, col)).all()
    G.close()


def test_iteration_limit(ptg, ctx):
    n, src, dst, s = chain(64, 7)
    off, col, w = csr(n, src, dst, True, 0)
    G = ctx.graph(off, col, w, symmetric=True)
    import ctypes
    o = ptg.RunOpts()
    out = np.empty(n, np.uint32)
    for limit, want in ((63, ptg.PTG_ERR_TIMEOUT), (64, ptg.PTG_OK)):
        o.max_iterations = limit
        assert ptg.lib().ptg_bfs(G.h, s, out.ctypes.data_as(ctypes.c_void_p), ctypes.byref(o)) == want
    assert sorted(out) == list(range(1, 65))


@functools.lru_cache(None)
def core_and_leaves(both_ways, seed):
    """A source joined to a complete core (8.7 M edges), and leaves on the core with degrees around the
    pull round's three ways to go over a row: the core is one frontier, and what it could still improve
    has far fewer edges.  Weights are the same both ways, or not on some edges."""
    rng = np.random.RandomState(seed)
    core = 2950
    degrees = np.concatenate([rng.randint(1, 17, 20011), rng.randint(17, 129, 500), rng.randint(129, 600, 60),
                              [15, 16, 17, 64, 65, 127, 128, 129, 255, 256, 257, 512, 513]])
    n = 1 + core + len(degrees) + 5  # five without edges
    a, b = np.meshgrid(np.arange(core), np.arange(core))
    keep = a < b
    src, dst = [np.zeros(core, np.int64), 1 + a[keep]], [1 + np.arange(core), 1 + b[keep]]
    leaf = np.repeat(np.arange(len(degrees)), degrees)
    src.append(1 + core + leaf)
    dst.append(1 + (leaf * 37 + np.arange(len(leaf)) * 3) % core)
    ids = rng.permutation(n)
    off, col, _ = csr(n, ids[np.concatenate(src)], ids[np.concatenate(dst)], True, 0)
    inv = np.argsort(ids)
    row = np.repeat(np.arange(n), np.diff(off).astype(np.int64))
    lo, hi = np.minimum(inv[row], inv[col]), np.maximum(inv[row], inv[col])
    h = (lo * 7919 + hi * 104729) % 61
    w = np.where(lo == 0, 5 + h % 2, np.where(hi <= core, 20 + h, 1 + h)).astype(np.uint32)
    if not both_ways:
        w += ((row < col) & (h < 9)).astype(np.uint32)
    return off, col, w, int(ids[0])


@pytest.mark.parametrize("both_ways", [True, False])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("grouped", [False, True])
def test_sssp_pull_rounds(ptg, ctx, ctx_grouped, oracle, grouped, wide, both_ways):
    off, col, w, s = core_and_leaves(both_ways, 11)
    G = (ctx_grouped if grouped else ctx).graph(off, col, w, symmetric=True, wide_offsets=wide)
    dist = oracle.sssp(off, col, w, s)
    for delta in (0, 3, 33, 1000000):
        st = {}
        assert (G.sssp(s, delta=delta, stats=st) == dist).all(), delta
        if delta == 1000000:  # (the core is one frontier)
            assert (st["bottom_up_rounds"] > 0) == both_ways
        assert (G.sssp(s, delta=delta, flags=ptg.PTG_NO_DIRECTION_OPT, stats=st) == dist).all(), delta
        assert st["bottom_up_rounds"] == 0
    G.close()


def test_buckets_beside_another_search(ptg, ctx, oracle):
    """Narrow buckets (a pass over the parked vertices per round or two) while another context's
    searches hold the same SMs, so that CTAs leave a barrier at very different times."""
    import threading
    cases = []
    for name in ("edge_degrees", "chain", "sparse", "large"):
        n, src, dst, s = GRAPHS[name]()
        off, col, w = csr(n, src, dst, True, n)
        cases.append((off, col, w, s, oracle.sssp(off, col, w, s)))
    other = ptg.Ctx(0)
    wrong, stop = [], threading.Event()

    def search(c, rounds):
        try:
            graphs = [c.graph(off, col, w, symmetric=True) for off, col, w, _, _ in cases]
            for r in range(rounds):
                if stop.is_set():
                    break
                for i, (g, case) in enumerate(zip(graphs, cases)):
                    for delta in (1, 7):
                        if not (g.sssp(case[3], delta=delta) == case[4]).all():
                            wrong.append((i, delta, r))
            for g in graphs:
                g.close()
        except Exception as e:
            wrong.append(repr(e))

    t = threading.Thread(target=search, args=(other, 1000))
    t.start()
    search(ctx, 10)
    stop.set()
    t.join()
    other.close()
    assert not wrong, wrong


@pytest.mark.parametrize("delta", [0xFFFFFFFD, 0xFFFFFFFE, 0xFFFFFFFF])
@pytest.mark.parametrize("zero_based", [False, True])
@pytest.mark.parametrize("name", ["edge_degrees", "sparse", "one_cta"])
@pytest.mark.parametrize("streamed", [False, True])
def test_bucket_width_past_every_distance(ptg, ctx, oracle, name, delta, zero_based, streamed):
    """Widths whose sum with the source's value reaches or passes 2^32: one bucket holds everything."""
    n, src, dst, s = GRAPHS[name]()
    off, col, w = csr(n, src, dst, not streamed, n)
    cfg = ptg.partition_config(partition_bytes=1024, device_budget_bytes=4096, force_out_of_core=1) if streamed else None
    G = ctx.graph(off, col, w, symmetric=not streamed, config=cfg)
    assert G.info()["out_of_core"] == int(streamed)
    dist = oracle.sssp(off, col, w, s)
    want = np.where(dist == 0xFFFFFFFF, dist, dist - 1) if zero_based else dist
    assert (G.sssp(s, delta=delta, flags=ptg.PTG_LEVEL_ZERO_BASED if zero_based else 0) == want).all()
    G.close()


@pytest.mark.parametrize("kind", ["bfs", "sssp", "cc"])
def test_barrier_wait_runs_out(ptg, oracle, kind):
    """Blocks that wait for the others at most one poll give up: the call reports a timeout, and the
    context answers the next call."""
    import ctypes
    n, src, dst, s = GRAPHS["large"]()
    off, col, w = csr(n, src, dst, True, n)
    c = ptg.Ctx(0)
    G = c.graph(off, col, w, symmetric=True)
    call = {"bfs": lambda: G.bfs(s), "sssp": lambda: G.sssp(s), "cc": lambda: G.cc(flags=ptg.PTG_REFERENCE_SCHEDULE)}[kind]
    want = {"bfs": lambda: oracle.bfs(off, col, s, method="queue"), "sssp": lambda: oracle.sssp(off, col, w, s),
            "cc": lambda: oracle.cc(off, col)}[kind]()
    polls = ptg.lib().ptg_internal_set_barrier_polls
    for _ in range(3):
        polls(c.h, ctypes.c_uint64(1))
        with pytest.raises(ptg.PtgError) as e:
            call()
        assert e.value.status == ptg.PTG_ERR_TIMEOUT
        assert "barrier" in str(e.value)
        polls(c.h, ctypes.c_uint64(1 << 26))
        assert (call() == want).all()
    c.close()


def test_long_searches_are_waited_for(ptg, oracle):
    """A search is one launch: the host's limit counts from its last sign of life, not from its start.
    (100 K levels, some 0.6 s, with a limit of 50 ms.)  Without any sign the call reports a timeout,
    and the context answers the next one."""
    import ctypes
    n, src, dst, s = chain(100000, 5)
    off, col, w = csr(n, src, dst, True, 0)
    c = ptg.Ctx(0)
    G = c.graph(off, col, w, symmetric=True)
    want = oracle.bfs(off, col, s, method="queue")
    wait = ptg.lib().ptg_internal_set_wait_ms
    assert (G.bfs(s) == want).all()
    wait(c.h, ctypes.c_uint32(50))
    assert (G.bfs(s) == want).all()
    assert (G.sssp(s, delta=1) == oracle.sssp(off, col, w, s)).all()
    wait(c.h, ctypes.c_uint32(0))
    with pytest.raises(ptg.PtgError) as e:
        G.bfs(s)
    assert e.value.status == ptg.PTG_ERR_TIMEOUT
    wait(c.h, ctypes.c_uint32(600000))
    assert (G.bfs(s) == want).all()
    c.close()
