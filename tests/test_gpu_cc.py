"""Connected components where the vertex-wise pass over the rows outside the
giant component can go wrong: rows at the edges of a warp's share and of a
queued piece, hubs with the smallest and with the largest id of their
component, empty and one-vertex graphs in a batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEGREES = [1, 2, 3, 4, 33, 1025, 1026, 1027, 2050, 2051, 5000]


def csr(n, src, dst):
    a = np.concatenate([src, dst]).astype(np.int64)
    b = np.concatenate([dst, src]).astype(np.int64)
    key = np.unique(a * n + b)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return off, (key % n).astype(np.uint32)


def star(deg, hub_first):
    hub = 0 if hub_first else deg
    leaves = np.array([v for v in range(deg + 1) if v != hub])
    return deg + 1, np.full(deg, hub), leaves


@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("hub_first", [False, True])
def test_components_outside_the_giant(ptg, ctx, ctx_grouped, oracle, grouped, wide, hub_first):
    rng = np.random.RandomState(3)
    big = 40001  # a random graph that the samples find as the giant, and its isolated vertices
    src, dst = [rng.randint(0, big, 120000)], [rng.randint(0, big, 120000)]
    n = big
    for d in DEGREES:
        k, s, t = star(d, hub_first)
        src.append(s + n)
        dst.append(t + n)
        n += k
    keep = np.concatenate(src) != np.concatenate(dst)
    off, col = csr(n, np.concatenate(src)[keep], np.concatenate(dst)[keep])
    c = ctx_grouped if grouped else ctx
    G = c.graph(off, col, symmetric=True, wide_offsets=wide)
    assert (G.cc() == oracle.cc(off, col, method="unionfind")).all()
    G.close()


@pytest.mark.parametrize("hub_first", [False, True])
def test_batch_of_stars_and_empty_graphs(ptg, ctx, oracle, hub_first):
    begin, n, src, dst = [0], 0, [np.zeros(0, int)], [np.zeros(0, int)]
    for d in DEGREES + [0, 0, 40, 0]:
        if d == 0:  # an empty graph, then one vertex without edges
            begin += [n, n + 1]
            n += 1
            continue
        k, s, t = star(d, hub_first)
        src.append(s + n)
        dst.append(t + n)
        n += k
        begin.append(n)
    off, col = csr(n, np.concatenate(src), np.concatenate(dst))
    whole = oracle.cc(off, col, method="unionfind").astype(np.int64)
    first = np.repeat(np.array(begin[:-1]), np.diff(begin))
    assert (ctx.cc_batch(np.array(begin, np.uint64), off, col) == whole - first).all()
