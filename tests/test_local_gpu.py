"""The per-source engine of low-degree graphs at the edges of its sizes: row widths 4, 8
and 16, levels around the row queue's 384 and 1536 vertices, the id queue's 6144 and the
rings' 8192 and 12288, graphs on both sides of the mesh form's sizes, and levels too wide
for any queue.  Distances and counts are integers and must equal the oracle's exactly."""
import numpy as np
import pytest

import gu
import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def check(hg, srcs):
    g = gu.Graph(hg)
    ref, _ = oracle.bfs_multi(hg.R, hg.C, hg.n, srcs, nthreads=8)
    reached = ref[ref != gu.UNREACHABLE]
    s = torch.as_tensor(np.asarray(srcs, np.int32), device="cuda")
    for _ in range(2):  # the second call finds what the first one's overflow left on the graph
        out = torch.full((len(srcs), hg.n), -7, dtype=torch.int32, device="cuda")
        g.bfs(s, out)
        np.testing.assert_array_equal(out.cpu().numpy(), ref)
        assert g.diameter(s) == reached.max()
        cnt = torch.full((len(srcs),), -1, dtype=torch.int64, device="cuda")
        g.reach(s, cnt)
        np.testing.assert_array_equal(cnt.cpu().numpy(), (ref != gu.UNREACHABLE).sum(1))


def fan(width, levels, out, step, seed):
    """A tree of out-degree `out` grown to exactly `width` leaves, then a ladder."""
    u, v, last, n = [], [], np.array([0]), 1
    while len(last) < width:
        m = min(width, len(last) * out)
        new = n + np.arange(m)
        u.append(last[np.arange(m) % len(last)])
        v.append(new)
        last, n = new, n + m
    for _ in range(levels):
        new = n + np.arange(width)
        for t in range(step):
            u.append(last)
            v.append(np.roll(new, -t))
        last, n = new, n + width
    u, v = np.concatenate(u), np.concatenate(v)
    p = np.random.default_rng(seed).permutation(n)
    return gu.HostGraph.from_edges(n, p[u], p[v], symmetric=False), int(p[0]), int(p[last[0]])


@pytest.mark.parametrize("width", [383, 384, 385, 1535, 1537, 4095, 4097, 6143, 6144, 6145, 8200])
@pytest.mark.parametrize("out,step", [(4, 1), (3, 3), (7, 7), (15, 2)])
def test_level_widths(width, out, step):
    hg, root, leaf = fan(width, 60, out, step, seed=width + out)
    check(hg, [root, leaf, root])


@pytest.mark.parametrize("side", [(1023, 1025), (1025, 1025), (724, 724), (725, 725), (33, 33), (1, 40000)])
def test_grids(side):
    """Graphs on both sides of the sizes at which the forms change."""
    hg = gu.HostGraph.grid(*side, seed=3)
    check(hg, gu.sources(hg.n, 5, seed=2))


def test_self_loops_double_edges_and_isolated_sources():
    rng = np.random.default_rng(5)
    n = 5000
    u = np.repeat(np.arange(n - 100), 2)
    v = np.where(rng.random(u.size) < 0.2, u, np.minimum(u + rng.integers(1, 40, u.size), n - 1))
    hg = gu.HostGraph.from_edges(n, u, v, symmetric=False)
    check(hg, [0, n - 1, 17, 17])


def test_every_id_of_a_large_graph():
    """Narrow levels over a million ids: those whose tag is the recent table's mark for an
    empty slot are claimed like the others."""
    hg, root, _ = fan(2000, 520, 7, 2, seed=8)
    check(hg, [root])
