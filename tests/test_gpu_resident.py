"""The one-launch traversal of in-HBM graphs at its edges: degrees around the
three work lists and a warp's pieces, one CTA and many, long chains (many
levels, many buckets), every offset width and vertex order, against the oracle."""
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
