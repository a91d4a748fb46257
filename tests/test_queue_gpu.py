"""gu_bfs_many's CTA groups: one item, a group per item of its own size, and more items
than half the grid's CTAs (equal groups and the counter), with requests split over
several items; rows and counts equal the oracle's exactly."""
import numpy as np
import pytest

import gu
import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graphs():
    hgs = [gu.HostGraph.rmat(8, 8, seed=1), gu.HostGraph.rmat(13, 16, seed=2), gu.HostGraph.dag(3000, 20000, seed=3),
           gu.HostGraph.grid(40, 30, 0.05, seed=4)]
    return [(hg, gu.Graph(hg)) for hg in hgs]


@pytest.mark.parametrize("items,kmax", [(1, 300), (2, 64), (5, 600), (40, 130), (151, 20), (152, 70), (153, 70), (400, 9)])
def test_items_and_groups(graphs, items, kmax):
    rng = np.random.default_rng(items)
    reqs, want = [], []
    for i in range(items):
        hg, g = graphs[i % len(graphs)]
        srcs = rng.integers(0, hg.n, int(rng.integers(1, kmax + 1))).astype(np.int32)
        s = torch.as_tensor(srcs, device="cuda")
        rows = torch.full((len(srcs), hg.n + 4 * (i % 2)), -7, dtype=torch.int32, device="cuda") if i % 3 != 2 else None
        cnt = torch.full((len(srcs),), -7, dtype=torch.int64, device="cuda") if i % 3 != 1 else None
        reqs.append((g, s, rows, cnt))
        want.append((hg, srcs))
    gu.bfs_many(reqs)
    for (g, s, rows, cnt), (hg, srcs) in zip(reqs, want):
        uniq, inv = np.unique(srcs, return_inverse=True)
        ref = oracle.bfs_multi(hg.R, hg.C, hg.n, uniq.astype(np.int32), nthreads=8)[0][inv]
        if rows is not None:
            got = rows.cpu().numpy()
            np.testing.assert_array_equal(got[:, : hg.n], ref)
            assert (got[:, hg.n:] == -7).all()
        if cnt is not None:
            np.testing.assert_array_equal(cnt.cpu().numpy(), (ref != gu.UNREACHABLE).sum(1))


@pytest.fixture(scope="module")
def trees():
    """Two trees on a million vertices: a slice of workspace for 64 sources is 0.23 GB."""
    n = 1 << 20
    return [gu.Graph(gu.HostGraph.from_edges(n, (np.arange(1, n) - 1) // f, np.arange(1, n))) for f in (16, 50)]


def test_workspace_on_large_graphs(trees):
    """As many slices of workspace as equal groups take (four here), however many requests."""
    srcs = torch.arange(7, 9, dtype=torch.int32, device="cuda")
    reqs = [(trees[i % 2], srcs, None, torch.zeros(2, dtype=torch.int64, device="cuda")) for i in range(32)]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    gu.bfs_many(reqs)
    assert free - torch.cuda.mem_get_info()[0] < 1.3e9
    for g, _, _, cnt in reqs:
        assert cnt.tolist() == [g.n, g.n]


def test_server_admits_what_equal_groups_take(trees):
    """Forty one-source requests on both graphs, merged into one launch or a few, within a
    budget of four slices and the outputs."""
    srv = gu.Server(hbm_budget_bytes=3 << 29, slots=1)
    out = [np.zeros(1, np.int64) for _ in range(40)]
    ids = [srv.submit(trees[i % 2], gu.QUERY_REACH, np.array([i], np.int32), out[i]) for i in range(40)]
    for i, rid in enumerate(ids):
        assert srv.wait(rid, 60.0) is not None
        assert out[i][0] == trees[i % 2].n
    srv.close()
