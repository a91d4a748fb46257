"""The shared-memory BFS engine (AUTO on small graphs and few sources) at the edges of
its sizes: word, slice and cluster boundaries, the byte form's last size, one CTA to
sixteen per source, wide and long searches.  Distances, counts and levels are
integers and must equal the oracle's exactly; the batched engine (GU_AUTO_LOCAL=0)
must give the same rows."""
import ctypes
import os

import numpy as np
import pytest

import gu
import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def rows(g, srcs, ld=None, batched=False):
    s = torch.as_tensor(np.asarray(srcs, np.int32), device="cuda")
    ld = g.n if ld is None else ld
    out = torch.full((len(srcs), ld), -7, dtype=torch.int32, device="cuda")
    if batched:
        os.environ["GU_AUTO_LOCAL"] = "0"
    try:
        g.bfs(s, out, ld=ld)
    finally:
        os.environ.pop("GU_AUTO_LOCAL", None)
    return out.cpu().numpy()


def hub_graph(n, m, seed, directed=False):
    """Random edges with a few hubs (out-degree above 512), so that AUTO never takes the
    low-degree engine and the whole-CTA expansion runs."""
    rng = np.random.default_rng(seed)
    u = rng.integers(0, n, m)
    v = rng.integers(0, n, m)
    hub = rng.integers(0, n, 2)
    u = np.concatenate([u, np.repeat(hub, min(n, 900))])
    v = np.concatenate([v, rng.integers(0, n, 2 * min(n, 900))])
    return gu.HostGraph.from_edges(n, u, v, symmetric=not directed)


def check(hg, srcs, ld=None):
    g = gu.Graph(hg)
    ref, _ = oracle.bfs_multi(hg.R, hg.C, hg.n, srcs, nthreads=8)
    got = rows(g, srcs, ld)
    td, bu, ml = g.last_launch()[1:]
    np.testing.assert_array_equal(got[:, : hg.n], ref)
    assert (got[:, hg.n:] == -7).all()
    reached = ref[ref != gu.UNREACHABLE]
    assert g.level_profile() == [] and ml == reached.max() and td + bu >= ml  # this engine ran
    np.testing.assert_array_equal(rows(g, srcs, batched=True), ref)
    s = torch.as_tensor(np.asarray(srcs, np.int32), device="cuda")
    cnt = torch.full((len(srcs),), -1, dtype=torch.int64, device="cuda")
    g.reach(s, cnt)
    np.testing.assert_array_equal(cnt.cpu().numpy(), (ref != gu.UNREACHABLE).sum(1))
    assert g.diameter(s) == reached.max()


@pytest.mark.parametrize("n,m,k", [(20, 100, 20), (31, 200, 3), (33, 200, 5), (1000, 9000, 400), (4097, 30000, 200),
                                   (8192, 50000, 20), (8193, 50000, 200), (16384, 90000, 1), (16384, 200000, 160),
                                   (16385, 150000, 30), (40001, 400000, 20), (65537, 500000, 3), (131073, 900000, 2),
                                   (262144, 1500000, 8)])
@pytest.mark.parametrize("directed", [False, True])
def test_sizes(n, m, k, directed):
    hg = hub_graph(n, m, seed=n + directed, directed=directed)
    check(hg, gu.sources(n, k, seed=5), ld=n + (n % 3))


def test_wide_levels_and_isolated_sources():
    """A star of 20,000 leaves (a level wider than the queue of 8192), duplicate sources,
    isolated vertices as sources."""
    n = 24000
    hg = gu.HostGraph.from_edges(n, np.zeros(20000, np.int32), np.arange(1, 20001))
    check(hg, np.array([0, 0, 5, 23999, 20001, 20000], np.int32))
    hg = gu.HostGraph.from_edges(12000, np.zeros(11990, np.int32), np.arange(1, 11991))
    check(hg, np.array([3, 0, 11999], np.int32))


def test_long_lists_and_long_paths():
    """Unvisited vertices with long in-lists outside the frontier (the warp's scan of what
    the first pieces leave), a full list of such vertices, and a path behind a hub."""
    rng = np.random.default_rng(3)
    n = 15000  # two dense halves joined by one edge: scans of the far half find nothing for a level
    a, b = rng.integers(0, n // 2, 500000), rng.integers(0, n // 2, 500000)
    c, d = rng.integers(n // 2, n, 500000), rng.integers(n // 2, n, 500000)
    hg = gu.HostGraph.from_edges(n, np.concatenate([a, c, [0]]), np.concatenate([b, d, [n - 1]]))
    check(hg, np.array([1, 77, n - 2], np.int32))
    path = np.arange(3000)
    hg = gu.HostGraph.from_edges(3100, np.concatenate([path[:-1], np.zeros(90, np.int64)]),
                                 np.concatenate([path[1:], np.arange(3000, 3090)]))
    check(hg, np.array([0, 1500, 2999, 3050], np.int32))


def test_levels_beyond_16_bits_rerun_on_the_batched_engine():
    n = 66000
    hg = gu.HostGraph.from_edges(n, np.concatenate([np.arange(n - 41), np.zeros(40, np.int64)]),
                                 np.concatenate([np.arange(1, n - 40), np.arange(n - 40, n)]))
    g = gu.Graph(hg)
    got = rows(g, [0])[0]
    np.testing.assert_array_equal(got[: n - 40], np.arange(n - 40))
    assert (got[n - 40:] == 1).all()


def test_bad_sources_and_other_streams():
    hg = hub_graph(9000, 60000, seed=2)
    g = gu.Graph(hg)
    ref, _ = oracle.bfs_multi(hg.R, hg.C, hg.n, [0, 4], nthreads=4)
    for bad in (hg.n, -1):
        s = torch.tensor([0, bad, 4], dtype=torch.int32, device="cuda")
        out = torch.full((3, hg.n), -7, dtype=torch.int32, device="cuda")
        with pytest.raises(gu.GuError) as e:
            g.bfs(s, out)
        assert e.value.status == 1
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        s = torch.tensor([0, 4], dtype=torch.int32, device="cuda")
        out = torch.empty((2, hg.n), dtype=torch.int32, device="cuda")
        g.bfs(s, out, stream=st)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)


def test_tuned_to_this_engine():
    hg = hub_graph(3000, 20000, seed=4)
    g = gu.Graph(hg)
    srcs = gu.sources(hg.n, 40, seed=1)
    ref, _ = oracle.bfs_multi(hg.R, hg.C, hg.n, srcs, nthreads=4)
    _, trials = g.autotune(torch.as_tensor(srcs, device="cuda"))
    assert "shared-memory" in {t["engine"] for t in trials}
    g.set_tuning({"engine": "shared-memory"})
    np.testing.assert_array_equal(rows(g, srcs), ref)


@pytest.mark.parametrize("n,k", [(198, 198), (3000, 300), (9000, 3), (20000, 7), (70000, 2)])
def test_refused_calls_write_nothing(n, k):
    """A source out of range, first or last: no row and no count is written, of the good
    sources neither (byte form, one CTA, clusters; BC and sigma too where they fit)."""
    hg = hub_graph(n, 9 * n, seed=n)
    g = gu.Graph(hg)
    for at, bad in ((0, n), (k - 1, -1)):
        srcs = gu.sources(n, k, seed=1)
        srcs[at] = bad
        s = torch.as_tensor(srcs, device="cuda")
        out = torch.full((k, n), -7, dtype=torch.int32, device="cuda")
        sig = torch.full((k, n), -7, dtype=torch.int64, device="cuda")
        delta = torch.full((k, n), -7.0, dtype=torch.float64, device="cuda")
        bc = torch.full((n,), -7.0, dtype=torch.float64, device="cuda")
        for call in (lambda: g.bfs(s, out), lambda: g.sigma(s, sig, dist_dev=out), lambda: g.bc(s, bc, delta_dev=delta)):
            with pytest.raises(gu.GuError) as e:
                call()
            assert e.value.status == 1
        for t in (out, sig, delta, bc):
            assert (t == -7).all()


@pytest.mark.parametrize("after", [0, 1])
@pytest.mark.parametrize("n", [900, 9000, 40000])
def test_without_memory_for_its_tables(n, after):
    """Its first (pinned) or second (device) allocation fails: the search runs on another
    engine, as on these graphs before this engine was there; a bad source is still
    refused, and the next call takes this engine."""
    hg = hub_graph(n, 8 * n, seed=n + after)
    srcs = gu.sources(n, 5, seed=2)
    ref, _ = oracle.bfs_multi(hg.R, hg.C, n, srcs, nthreads=4)
    L = gu.lib()
    L.gu_debug_fail_allocations.argtypes = [ctypes.c_int64, ctypes.c_int64]
    s = torch.as_tensor(srcs, device="cuda")
    for what in ("bfs", "reach", "diameter", "bad source"):
        g = gu.Graph(hg)
        cnt = torch.full((5,), -1, dtype=torch.int64, device="cuda")
        out = torch.full((5, n), -7, dtype=torch.int32, device="cuda")
        try:
            assert L.gu_debug_fail_allocations(after, 1) == gu.OK
            if what == "bfs":
                g.bfs(s, out)
                np.testing.assert_array_equal(out.cpu().numpy(), ref)
            elif what == "reach":
                g.reach(s, cnt)
                np.testing.assert_array_equal(cnt.cpu().numpy(), (ref != gu.UNREACHABLE).sum(1))
            elif what == "diameter":
                assert g.diameter(s) == ref[ref != gu.UNREACHABLE].max()
            else:
                with pytest.raises(gu.GuError) as e:
                    g.bfs(torch.tensor([1, n], dtype=torch.int32, device="cuda"), out[:2])
                assert e.value.status == 1
        finally:
            L.gu_debug_fail_allocations(0, 0)
        np.testing.assert_array_equal(rows(g, srcs), ref)
        assert g.level_profile() == []


def test_direction_counts_all_frontier_edges():
    """1024 neighbours of the source, in the first words of the bitmap, with 64 out-edges
    each: their edges are summed by other warps than find them, and all 65536 count.  The
    second level is then searched bottom-up (65536^2 against twice 6975 vertices left x
    200000 edges) and finds all of them, and so is the third, which finds nothing; with
    part of the edges the second would be top-down, as the first is."""
    rng = np.random.default_rng(4)
    n, mid, end = 16000, 1025, 8000
    u = np.concatenate([np.zeros(1024, np.int64), np.repeat(np.arange(1, mid), 64), rng.integers(mid, end, 133440)])
    v = np.concatenate([np.arange(1, mid), rng.integers(mid, end, 65536), rng.integers(mid, end, 133440)])
    order = np.argsort(u, kind="stable")  # parallel edges stay: the counts are exact
    R = np.concatenate([[0], np.cumsum(np.bincount(u, minlength=n))])
    hg = gu.HostGraph(R, v[order], n, directed=True)
    g = gu.Graph(hg)
    got = rows(g, [0])
    td, bu, ml = g.last_launch()[1:]
    np.testing.assert_array_equal(got, oracle.bfs_multi(hg.R, hg.C, n, [0])[0])
    assert g.level_profile() == [] and (td, bu, ml) == (1, 2, 2)
