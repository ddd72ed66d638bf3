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


def test_level_masks_are_given_back(ptg):
    """What a call of 256 sources kept its levels in (12 x 32 MB here) is free for others after it."""
    torch = pytest.importorskip("torch")
    n, k = 1 << 20, 256
    rng = np.random.RandomState(1)
    key = np.unique(rng.randint(0, n, 1 << 22).astype(np.int64) * n + rng.randint(0, n, 1 << 22))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    c = ptg.Ctx(0)
    G = c.graph(off, (key % n).astype(np.uint32))
    out = torch.empty((k, n), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    before = c.device_info()["free_bytes"]
    G.msbfs(rng.randint(0, n, k).astype(np.uint32), flags=ptg.PTG_OUT_DEVICE, out=out)
    kept = before - c.device_info()["free_bytes"]
    assert kept < 3 * 32 * n + (64 << 20)  # a level, the next and the seen mask, queues and scans
    c.close()


@pytest.mark.parametrize("masks", [0, 1, 3, 5, 30])
def test_served_batches_fit_the_budget(ptg, oracle, masks):
    """A lane's batches are sized by the three masks that a level needs, and keep as many levels
    as the budget has room for besides."""
    n, k = 1 << 14, 256
    off, col, _ = chain_with_leaves(40, n, 3)
    m = col.size
    need = 3 * 32 * n + 4 * k * n + 8 * n + 16 * (n + 1) + 4 * (m // 2048 + 4)
    c = ptg.Ctx(0)
    G = c.graph(off, col, symmetric=True)
    assert not G.info()["degree_grouped"]
    srv = ptg.Server(c, lanes=1, max_slots=2 * k, memory_budget_bytes=need + masks * 32 * n + 64)
    gid = srv.add_graph(G)
    srcs = [int(s) for s in np.random.RandomState(masks).randint(0, n, 600)]
    ids = [srv.submit(gid, ptg.PTG_Q_BFS, s) for s in srcs]
    rows = [srv.wait(i)[0] for i in ids]
    st = srv.stats()
    assert st["max_batch_seen"] == k
    for s, row in list(zip(srcs, rows))[::20]:
        assert (row == oracle.bfs(off, col, s, method="queue")).all()
    c.close()


@pytest.mark.parametrize("out_weights,back_weights", [
    ((158294597, 252129289, 84674016, 232866233), (169702344, 154819396, 62669269, 58675956)),
    ((251776810, 242173211, 73729864, 188310061), (19052126, 157150182, 155272291, 72500844)),
])
def test_weights_chosen_to_look_symmetric(ptg, ctx, oracle, out_weights, back_weights):
    """A star whose edges weigh something else outwards than back, with weights for which the sums
    of an unkeyed hash agree: its rounds must not take the one for the other."""
    off = np.array([0, 4, 5, 6, 7, 8], np.uint64)
    col = np.array([1, 2, 3, 4, 0, 0, 0, 0], np.uint32)
    w = np.array(out_weights + back_weights, np.uint32)
    G = ctx.graph(off, col, w, symmetric=True)
    for s in range(5):
        assert (G.mssssp(np.array([s], np.uint32))[0] == oracle.sssp(off, col, w, s)).all()
    G.close()
