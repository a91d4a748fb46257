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
