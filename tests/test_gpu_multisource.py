"""Multi-source passes at their edges: source counts around the mask words,
searches with fewer, as many and more levels than the level history keeps, and
both vertex orders, against the oracle row by row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain_with_leaves(length, n, seed):
    """A path of `length` vertices and leaves hung on random vertices of it; every 7th vertex isolated."""
    rng = np.random.RandomState(seed)
    ids = rng.permutation(n)
    path, rest = ids[:length], ids[length:]
    rest = rest[np.arange(rest.size) % 7 != 0]
    src = np.concatenate([path[:-1], rest])
    dst = np.concatenate([path[1:], path[rng.randint(0, length, rest.size)]])
    a, b = np.concatenate([src, dst]), np.concatenate([dst, src])
    key = np.unique(a.astype(np.int64) * n + b)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    col = (key % n).astype(np.uint32)
    row = key // n
    w = (1 + (np.minimum(row, key % n) * 31 + np.maximum(row, key % n)) % 63).astype(np.uint32)
    return off, col, w


@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("length,n,k", [(2, 33, 1), (6, 100, 63), (7, 257, 64), (9, 500, 65), (11, 1001, 128),
                                        (12, 1002, 128), (13, 1003, 129), (24, 1200, 7), (40, 2049, 255), (40, 2050, 256)])
def test_levels_kept_and_written(ptg, ctx, ctx_grouped, oracle, grouped, wide, length, n, k):
    off, col, w = chain_with_leaves(length, n, length)
    c = ctx_grouped if grouped else ctx
    G = c.graph(off, col, w, symmetric=True, wide_offsets=wide)
    srcs = np.random.RandomState(k).randint(0, n, k).astype(np.uint32)
    rows, dist = G.msbfs(srcs), G.mssssp(srcs)
    known = {}
    for i, s in enumerate(srcs):
        s = int(s)
        if s not in known:
            known[s] = oracle.bfs(off, col, s, method="queue"), oracle.sssp(off, col, w, s)
        assert (rows[i] == known[s][0]).all()
        assert (dist[i] == known[s][1]).all()
    G.close()


@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("both_ways", [True, False])
@pytest.mark.parametrize("n,m,k", [(300, 4000, 64), (2001, 9000, 5), (5000, 400000, 64)])
def test_dense_sssp_rounds(ptg, ctx, ctx_grouped, oracle, grouped, both_ways, n, m, k):
    """Rounds over most of the edges, with the same weight both ways (they may
    be pulled) and with a weight of its own on every directed edge (they may
    not), rows around the pull split, a second component and large weights."""
    rng = np.random.RandomState(n)
    a, b = rng.randint(0, n - 40, m), (rng.randint(0, n - 40, m) * rng.randint(0, 2, m)) // 2
    a, b = np.concatenate([a, np.full(33, n - 1)]), np.concatenate([b, n - 2 - np.arange(33)])
    keep = a != b
    a, b = a[keep], b[keep]
    key = np.unique(np.concatenate([a, b]).astype(np.int64) * n + np.concatenate([b, a]))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    row, col = key // n, key % n
    mix = np.minimum(row, col) * 7919 + np.maximum(row, col) * 31 if both_ways else row * 7919 + col * 31
    w = np.where(mix % 97 == 0, 1 << 29, mix % 64).astype(np.uint32)
    G = (ctx_grouped if grouped else ctx).graph(off, col.astype(np.uint32), w, symmetric=True)
    srcs = rng.randint(0, n, k).astype(np.uint32)
    srcs[0] = n - 1
    dist = G.mssssp(srcs)
    for i, s in enumerate(srcs):
        assert (dist[i] == oracle.sssp(off, col.astype(np.uint32), w, int(s))).all()
    G.close()
