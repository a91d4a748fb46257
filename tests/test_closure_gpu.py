"""gu_dag_reach on bit rows at the edges of its chunks (4096 columns), column blocks
(512 MiB of rows) and level structure, against the oracle's per-vertex set sizes.
Counts are integers: the comparisons are exact."""
import ctypes

import numpy as np
import pytest

import gu
import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def closure(hg, stream=None):
    g = gu.Graph(hg)
    cnt = torch.full((max(hg.n, 1),), -5, dtype=torch.int64, device="cuda")
    tot = g.dag_reach(cnt[: hg.n], stream=stream)
    again = torch.full((max(hg.n, 1),), -7, dtype=torch.int64, device="cuda")
    assert g.dag_reach(again[: hg.n]) == tot  # the kept order, a second time
    np.testing.assert_array_equal(cnt.cpu().numpy()[: hg.n], again.cpu().numpy()[: hg.n])
    return cnt.cpu().numpy()[: hg.n], tot


@pytest.mark.parametrize("n,m", [(1, 0), (2, 1), (31, 60), (4095, 9000), (4096, 30000), (4097, 30000), (8193, 2000),
                                 (70001, 280000)])
def test_sizes_vs_oracle(n, m):
    rng = np.random.default_rng(n)
    a, b = rng.integers(0, n, m), rng.integers(0, n, m)
    keep = a != b
    perm = rng.permutation(n)
    hg = gu.HostGraph.from_edges(n, perm[np.minimum(a, b)[keep]], perm[np.maximum(a, b)[keep]], symmetric=False)
    counts, tot = closure(hg)
    ref, rtot = oracle.dag_reach_counts(hg.R, hg.C, hg.n)
    np.testing.assert_array_equal(counts, ref)
    assert tot == rtot


def test_path_star_and_empty():
    n = 5000
    path = gu.HostGraph.from_edges(n, np.arange(n - 1), np.arange(1, n), symmetric=False)  # 5000 levels
    counts, tot = closure(path)
    np.testing.assert_array_equal(counts, np.arange(n - 1, -1, -1))
    star = gu.HostGraph.from_edges(n, np.zeros(n - 1, np.int32), np.arange(1, n), symmetric=False)  # one hub
    counts, tot = closure(star)
    assert tot == n - 1 and counts[0] == n - 1 and not counts[1:].any()
    counts, tot = closure(gu.HostGraph(np.zeros(11, np.int32), np.zeros(0, np.int32), 10, True))
    assert tot == 0 and not counts.any()


def test_cycles_and_self_loops_keep_the_search():
    """A directed graph with a cycle has no topological order: the counts are still the
    numbers of other vertices reached, as the search from every vertex gives them."""
    hg = gu.HostGraph.from_edges(300, np.arange(300), (np.arange(300) + 1) % 300, symmetric=False)
    counts, tot = closure(hg)
    assert tot == 300 * 299 and (counts == 299).all()
    R = np.array([0, 2, 3, 3], np.int32)  # 0 -> 0, 0 -> 1, 1 -> 2
    counts, tot = closure(gu.HostGraph(R, np.array([0, 1, 2], np.int32), 3, True))
    np.testing.assert_array_equal(counts, [2, 1, 0])


def test_no_memory_for_rows_falls_back():
    hg = gu.HostGraph.dag(3000, 24000, seed=1)
    ref, rtot = oracle.dag_reach_counts(hg.R, hg.C, hg.n)
    g = gu.Graph(hg)
    cnt = torch.empty(hg.n, dtype=torch.int64, device="cuda")
    fail = gu.lib().gu_debug_fail_allocations
    fail.argtypes = [ctypes.c_int64, ctypes.c_int64]
    try:
        # io staging, plan scratch and the order fit; both tries for the rows fail
        assert fail(3, 2) == gu.OK
        assert g.dag_reach(cnt) == rtot
    finally:
        fail(0, 0)
    np.testing.assert_array_equal(cnt.cpu().numpy(), ref)
    assert g.dag_reach(cnt) == rtot
    np.testing.assert_array_equal(cnt.cpu().numpy(), ref)


@pytest.mark.parametrize("n,m,k", [(16385, 60000, 5), (17001, 90000, 64), (20011, 100000, 65), (30000, 120000, 128),
                                   (40000, 300000, 129), (70001, 280000, 256), (50000, 50000, 600)])
def test_reach_by_levels_vs_search(n, m, k, monkeypatch):
    """gu_reach on an acyclic graph (rows of source bits, level by level): counts equal
    the oracle's and the batched search's at every row width and across batches, with
    duplicate and sink sources."""
    rng = np.random.default_rng(n)
    a, b = rng.integers(0, n, m), rng.integers(0, n, m)
    keep = a != b
    perm = rng.permutation(n)
    hub = perm[n - 1]  # one vertex with a long in-list
    u = np.concatenate([perm[np.minimum(a, b)[keep]], perm[:1500]])
    v = np.concatenate([perm[np.maximum(a, b)[keep]], np.full(1500, hub)])
    hg = gu.HostGraph.from_edges(n, u, v, symmetric=False)
    g = gu.Graph(hg)
    srcs = gu.sources(n, k, seed=4)
    srcs[:3] = [perm[n - 1], perm[0], perm[0]]
    s = torch.as_tensor(srcs, device="cuda")
    cnt = torch.full((k,), -1, dtype=torch.int64, device="cuda")
    g.reach(s, cnt)  # the first call searches, the next ones have the order
    first = cnt.cpu().numpy()
    for _ in range(2):
        cnt.fill_(-1)
        g.reach(s, cnt)
        np.testing.assert_array_equal(cnt.cpu().numpy(), first)
    assert g.level_profile() == []  # no search ran
    got = cnt.cpu().numpy()
    monkeypatch.setenv("GU_AUTO_LOCAL", "0")
    g.reach(s, cnt)
    np.testing.assert_array_equal(got, cnt.cpu().numpy())
    some = list(range(0, k, max(1, k // 6)))
    ref, _ = oracle.bfs_multi(hg.R, hg.C, n, srcs[some], nthreads=8)
    np.testing.assert_array_equal(got[some], (ref != gu.UNREACHABLE).sum(1))


def test_reach_on_deep_and_cyclic_graphs():
    n = 20000
    chain = gu.HostGraph.from_edges(n, np.arange(n - 1), np.arange(1, n), symmetric=False)  # too many levels
    ring = gu.HostGraph.from_edges(n, np.arange(n), (np.arange(n) + 1) % n, symmetric=False)  # a cycle
    s = torch.arange(0, n, 2500, dtype=torch.int32, device="cuda")
    for hg, want in ((chain, n - np.arange(0, n, 2500)), (ring, np.full(8, n))):
        g = gu.Graph(hg)
        for _ in range(3):
            cnt = torch.full((8,), -1, dtype=torch.int64, device="cuda")
            g.reach(s, cnt)
            np.testing.assert_array_equal(cnt.cpu().numpy(), want)


@pytest.mark.parametrize("levels", [96, 97, 5000])
def test_orders_that_are_not_used_are_not_kept(levels):
    """Reachable counts go by orders of up to 96 levels.  A deeper one is not built for them,
    nor anything kept of it or of a graph with a cycle; the closure still builds it, and
    the counts are the same throughout."""
    n = 20000
    v = np.arange(n)
    u = v[(v % levels != levels - 1) & (v < n - 1)]
    ends = np.setdiff1d(v, u)[:20] if levels < 1000 else np.full(20, n - 1) - np.arange(20)
    # (a hub in front of some vertices, so that the graph is not one of low out-degree)
    chains = gu.HostGraph.from_edges(n + 1, np.concatenate([u, np.full(20, n)]), np.concatenate([u + 1, ends]), symmetric=False)
    ring = gu.HostGraph.from_edges(n, v, (v + 1) % n, symmetric=False)
    order_bytes = 4 * (6 * n + 3 + 2 * (n - n // levels - 1))
    s = torch.arange(0, n, 2501, dtype=torch.int32, device="cuda")
    at = s.cpu().numpy()
    to_end = np.minimum(levels - 1 - at % levels, n - 1 - at) + 1  # a chain's vertices from each source on
    for hg, want in ((chains, to_end), (ring, np.full(len(at), n))):
        g = gu.Graph(hg)
        cnt = torch.full((len(at),), -1, dtype=torch.int64, device="cuda")

        def counts_are_right():
            g.reach(s, cnt)
            np.testing.assert_array_equal(cnt.cpu().numpy(), want)

        counts_are_right()
        before = g.device_bytes()
        for _ in range(3):
            counts_are_right()
        kept = g.device_bytes() - before  # and what the workspace grew by, at most 0.35 MB here
        assert (kept >= order_bytes) == (hg is chains and levels <= 96)
        sizes = torch.empty(hg.n, dtype=torch.int64, device="cuda")
        g.dag_reach(sizes)
        np.testing.assert_array_equal(sizes.cpu().numpy()[at], want - 1)
        if hg is ring:  # the search's workspace, not the closure's rows (50 MB)
            assert g.device_bytes() - before < 10e6
        counts_are_right()


def test_low_degree_graphs_stay_with_the_search():
    """Trees and graphs of few vertices per level, out-degree up to 16: no order is built
    for their reachable counts; one of many vertices per level has one from the second
    call on.  The counts are right either way."""
    n = 20000
    i = np.arange(1, n)
    rng = np.random.default_rng(3)
    layers = [np.concatenate([l * 200 + np.repeat(np.arange(200), 4) for l in range(90)]),
              np.concatenate([(l + 1) * 200 + rng.integers(0, 200, 800) for l in range(90)])]
    wide = [np.repeat(np.arange(15000), 5), 15000 + rng.integers(0, 5000, 75000)]
    for u, v, ordered in (((i - 1) // 2, i, False), (layers[0], layers[1], False), (wide[0], wide[1], True)):
        hg = gu.HostGraph.from_edges(n, u, v, symmetric=False)
        g = gu.Graph(hg)
        srcs = gu.sources(n, 9, seed=1)
        s = torch.as_tensor(srcs, device="cuda")
        want = (oracle.bfs_multi(hg.R, hg.C, n, srcs)[0] != gu.UNREACHABLE).sum(1)
        cnt = torch.full((9,), -1, dtype=torch.int64, device="cuda")
        sizes = []
        for _ in range(3):
            g.reach(s, cnt)
            np.testing.assert_array_equal(cnt.cpu().numpy(), want)
            sizes.append(g.device_bytes())
        # the order is 24 bytes a vertex and 8 an edge; the workspace grows by less here
        assert (sizes[2] - sizes[0] >= 24 * n + 8 * hg.m) == ordered


@pytest.mark.parametrize("n", [3000, 9000])
def test_stars_and_hubs(n):
    """A hub's successors are ORed one after another: a graph that is little else goes to
    the search from every vertex; the sizes are the same either way."""
    i = np.arange(1, n)
    for u, v in ((i * 0, i), (np.concatenate([i * 0, i[:-1]]), np.concatenate([i, i[1:]])), (i * 0, i // 2 * 2)):
        keep = u != v
        hg = gu.HostGraph.from_edges(n, u[keep], v[keep], symmetric=False)
        counts, tot = closure(hg)
        ref, rtot = oracle.dag_reach_counts(hg.R, hg.C, hg.n)
        np.testing.assert_array_equal(counts, ref)
        assert tot == rtot
