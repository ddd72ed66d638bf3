"""Streamed graphs whose rounds read host memory in place: rows over several
partitions, sparse and dense rounds, each way the host arrays can lie and each
placement, against the oracle."""
import numpy as np
import pytest

from test_gpu_resident import chain, csr, hubs, random_graph

pytestmark = pytest.mark.gpu

GRAPHS = {
    "rows_over_partitions": lambda: hubs([1, 16, 129, 1023, 1024, 1025, 9000], 1),
    "chain": lambda: chain(500, 2),
    "dense": lambda: random_graph(1999, 300000, 5),
    "large": lambda: random_graph(100003, 900000, 6),
}


@pytest.mark.parametrize("name", GRAPHS)
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("host", ["pinned", "pageable"])
@pytest.mark.parametrize("policy", ["PREFIX", "NONE", "HOT"])
def test_streamed_traversals_match_oracle(ptg, ctx, oracle, name, wide, host, policy):
    torch = pytest.importorskip("torch")
    n, src, dst, s = GRAPHS[name]()
    off, col, w = csr(n, src, dst, True, n)
    keep = None
    if host == "pinned":
        keep = [torch.from_numpy(a.view(np.int32)).pin_memory() for a in (col, w)]
        col, w = [a.numpy().view(np.uint32) for a in keep]
    m = col.size
    cfg = ptg.partition_config(partition_bytes=8192, device_budget_bytes=max(3 * 8192, m * 8 // 3), force_out_of_core=1,
                               hot_threshold=1, resident_policy=getattr(ptg, "PTG_RESIDENT_" + policy))
    G = ctx.graph(off, col, w, symmetric=False, config=cfg, wide_offsets=wide, pinned=host == "pinned")
    assert G.info()["out_of_core"] == 1
    st = {}
    assert (G.bfs(s, stats=st) == oracle.bfs(off, col, s, method="queue")).all()
    if name == "chain" and policy == "NONE" and host == "pinned":  # one vertex a round: its edges, not its partition
        assert st["link_bytes"] <= 4 * m
    dist = oracle.sssp(off, col, w, s)
    for delta in (0, 9):
        assert (G.sssp(s, delta=delta) == dist).all()
    assert (G.cc() == oracle.cc(off, col)).all()
    G.close()


@pytest.mark.parametrize("slots", [3, 64])
@pytest.mark.parametrize("host", ["pinned", "pageable"])
def test_sparse_rounds_fill_the_hot_cache(ptg, ctx, oracle, slots, host):
    """PTG_RESIDENT_HOT where every round reads one vertex's edges: the partitions are promoted by
    their visits all the same, so the next search needs less of the link (11 of 12 have a slot at most)."""
    torch = pytest.importorskip("torch")
    n, src, dst, s = chain(6000, 3)
    off, col, w = csr(n, src, dst, True, n)
    keep = None
    if host == "pinned":
        keep = [torch.from_numpy(a.view(np.int32)).pin_memory() for a in (col, w)]
        col, w = [a.numpy().view(np.uint32) for a in keep]
    cfg = ptg.partition_config(partition_bytes=8192, device_budget_bytes=(slots + 2) * 8192, force_out_of_core=1,
                               hot_threshold=3600, resident_policy=ptg.PTG_RESIDENT_HOT)
    G = ctx.graph(off, col, w, symmetric=False, config=cfg, pinned=host == "pinned")
    assert G.info()["partitions"] == 12
    dist = oracle.sssp(off, col, w, s)
    first, second = {}, {}
    assert (G.sssp(s, stats=first) == dist).all()
    assert (G.sssp(s, stats=second) == dist).all()
    assert second["partitions_cached"] > 0
    assert second["link_bytes"] < first["link_bytes"]
    if slots == 64:
        assert second["link_bytes"] * 5 < first["link_bytes"]
    G.close()


@pytest.mark.parametrize("shift", [(0, 0), (1, 0), (0, 1023), (700, 3)])
@pytest.mark.parametrize("policy", ["PREFIX", "NONE"])
@pytest.mark.parametrize("name,length", [("chain", 20000), ("hubs", 0)])
def test_ends_that_cannot_be_page_locked(ptg, ctx, oracle, shift, policy, name, length):
    """Pageable arrays that begin and end somewhere in a page: the edges of the partial pages are read
    in place as well, from the first and last partition too."""
    n, src, dst, s = chain(length, 4) if length else hubs([5000, 9000, 20000, 40000], 2)
    off, col, w = csr(n, src, dst, True, n)
    m = col.size

    def place(a, at):
        room = np.zeros(m + (1 << 15) + at, np.uint32)  # (of its own: no page shared with another array)
        first = -(room.ctypes.data // 4) % (1 << 14) + at  # `at` words behind a 64 KB boundary
        room[first:first + m] = a
        return room[first:first + m]

    col, w = place(col, shift[0]), place(w, shift[1])
    cfg = ptg.partition_config(partition_bytes=1 << 15, device_budget_bytes=3 << 15, force_out_of_core=1,
                               resident_policy=getattr(ptg, "PTG_RESIDENT_" + policy))
    G = ctx.graph(off, col, w, symmetric=False, config=cfg)
    st = {}
    assert (G.bfs(s, stats=st) == oracle.bfs(off, col, s, method="queue")).all()
    if name == "chain":  # a vertex a round: its edges, not its partition
        assert st["link_bytes"] <= 4 * m
    assert (G.sssp(s, stats=st) == oracle.sssp(off, col, w, s)).all()
    if name == "chain":
        assert st["link_bytes"] <= 8 * m
    else:
        assert (G.cc() == oracle.cc(off, col)).all()
    G.close()
