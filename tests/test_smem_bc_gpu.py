"""gu_bc and gu_sigma on small graphs (one CTA per source, state in shared memory) at the
edges of their sizes and list lengths: counts and distances exact, dependencies and
betweenness within 1e-12 relative of the FP64 oracle, equal bits on a second call."""
import numpy as np
import pytest

import gu
import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
RTOL = 1e-12


def check(hg, srcs, directed=False):
    g = gu.Graph(hg)
    n, k = hg.n, len(srcs)
    s = torch.as_tensor(np.asarray(srcs, np.int32), device="cuda")
    sig = torch.full((k, n), -7, dtype=torch.int64, device="cuda")
    d = torch.full((k, n), -7, dtype=torch.int32, device="cuda")
    g.sigma(s, sig, dist_dev=d)
    assert g.level_profile() == []  # no phase timeline: this engine ran
    rd, rs = oracle.sigma_multi(hg.R, hg.C, n, srcs, nthreads=8)
    np.testing.assert_array_equal(d.cpu().numpy(), rd)
    np.testing.assert_array_equal(sig.cpu().numpy().view(np.uint64), rs)
    bc = torch.empty(n, dtype=torch.float64, device="cuda")
    delta = torch.full((k, n), -7.0, dtype=torch.float64, device="cuda")
    g.bc(s, bc, delta_dev=delta)
    assert g.last_launch()[3] == rd[rd != gu.UNREACHABLE].max()
    again = torch.empty_like(bc)
    g.bc(s, again)
    assert torch.equal(bc.view(torch.int64), again.view(torch.int64))
    np.testing.assert_allclose(bc.cpu().numpy(), oracle.bc(hg.R, hg.C, n, srcs, pull=directed, nthreads=8), rtol=RTOL, atol=0)
    for i in range(0, k, max(1, k // 8)):
        _, _, ref = oracle.brandes(hg.R, hg.C, n, int(srcs[i]), "pull" if directed else "f64")
        np.testing.assert_allclose(delta[i].cpu().numpy(), ref, rtol=RTOL, atol=0)


@pytest.mark.parametrize("n,m,k", [(2, 1, 2), (7, 12, 7), (33, 300, 33), (64, 2000, 64), (1023, 8000, 200), (1025, 30000, 700),
                                   (4097, 150000, 40), (8191, 40000, 300), (8192, 400000, 20)])
@pytest.mark.parametrize("directed", [False, True])
def test_sizes(n, m, k, directed):
    rng = np.random.default_rng(n + directed)
    u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    if n > 1000:  # hubs: lists of a few entries up to thousands in one level
        hub = rng.integers(0, n, 3)
        u = np.concatenate([u, np.repeat(hub, 700)])
        v = np.concatenate([v, rng.integers(0, n, 2100)])
    hg = gu.HostGraph.from_edges(n, u, v, symmetric=not directed)
    check(hg, gu.sources(n, k, seed=3), directed)


def test_shapes():
    path = gu.HostGraph.from_edges(900, np.arange(899), np.arange(1, 900))  # 900 levels of one vertex
    check(path, np.array([0, 450, 899], np.int32))
    star = gu.HostGraph.from_edges(8000, np.zeros(7990, np.int32), np.arange(1, 7991))  # one list of 7990, isolated ends
    check(star, np.array([0, 5, 7999, 5], np.int32))
    # complete bipartite layers: lists of 63, 64 and 65 successors at every level
    for w in (32, 63, 64, 65):
        a, b = np.meshgrid(np.arange(w), np.arange(w))
        u = np.concatenate([(l * w + a).ravel() for l in range(5)])
        v = np.concatenate([((l + 1) * w + b).ravel() for l in range(5)])
        check(gu.HostGraph.from_edges(6 * w, u, v), np.arange(0, 6 * w, 11, dtype=np.int32))


def test_counts_wrap_and_wide_ranges():
    """8-wide complete layers: 8^(l - 1) paths to level l, past 2^64 (the counts wrap, as
    the oracle's do); with 12 layers the successors' terms span 2^33 and the
    dependencies still agree."""
    a, b = np.meshgrid(np.arange(8), np.arange(8))
    for layers in (30, 12):
        u = np.concatenate([(l * 8 + a).ravel() for l in range(layers - 1)] + [np.full(8, 8 * layers - 1), [0]])
        v = np.concatenate([((l + 1) * 8 + b).ravel() for l in range(layers - 1)] + [np.arange(8) + 8 * layers, [8 * layers]])
        hg = gu.HostGraph.from_edges(8 * layers + 8, u, v)
        if layers == 12:
            check(hg, np.arange(0, hg.n, 5, dtype=np.int32))
            continue
        g = gu.Graph(hg)
        s = torch.tensor([0, 3, 100], dtype=torch.int32, device="cuda")
        sig = torch.empty((3, hg.n), dtype=torch.int64, device="cuda")
        g.sigma(s, sig)
        _, rs = oracle.sigma_multi(hg.R, hg.C, hg.n, np.array([0, 3, 100], np.int32))
        np.testing.assert_array_equal(sig.cpu().numpy().view(np.uint64), rs)


def test_bad_sources_and_batches():
    hg = gu.HostGraph.rmat(9, 8, seed=1)
    g = gu.Graph(hg)
    bc = torch.full((hg.n,), -7.0, dtype=torch.float64, device="cuda")
    sig = torch.empty((2, hg.n), dtype=torch.int64, device="cuda")
    for bad in (hg.n, -1):
        s = torch.tensor([0, bad], dtype=torch.int32, device="cuda")
        for call in (lambda: g.bc(s, bc), lambda: g.sigma(s, sig)):
            with pytest.raises(gu.GuError) as e:
                call()
            assert e.value.status == 1
        assert (bc == -7.0).all()
    s = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    for batch in (100, 192):
        with pytest.raises(gu.GuError) as e:
            g.bc(s, bc, batch=batch)
        assert e.value.status == 1
    srcs = gu.sources(hg.n, 200, seed=2)
    s = torch.as_tensor(srcs, device="cuda")
    ref = oracle.bc(hg.R, hg.C, hg.n, srcs, nthreads=4)
    for batch in (0, 64, 256):  # 64: passes, the batched engine
        g.bc(s, bc, batch=batch)
        assert (g.level_profile() == []) == (batch != 64)
        np.testing.assert_allclose(bc.cpu().numpy(), ref, rtol=RTOL, atol=0)


def test_parallel_edges_on_few_vertices():
    """Lists longer than the graph has vertices (parallel edges are kept): those of 64
    entries and more come first in a level whatever n is, so that no lane sums a list
    longer than its integer sum has room for."""
    n, rng = 40, np.random.default_rng(9)
    # layers 0 | 1 .. 20 | 21 .. 39: lists of 40 .. 60 and of 300 entries in one level, the
    # longer ones behind
    reps = np.where(np.arange(20) % 3 == 2, 300, rng.integers(40, 60, 20))
    R = np.zeros(n + 1, np.int32)
    lists = [np.arange(1, 21)] + [np.sort(rng.integers(21, 40, r)) for r in reps] + [np.zeros(0, np.int64)] * 19
    R[1:] = np.cumsum([len(x) for x in lists])
    hg = gu.HostGraph(R, np.concatenate(lists).astype(np.int32), n, directed=True)
    check(hg, np.resize(np.arange(n, dtype=np.int32), 640), directed=True)


@pytest.mark.parametrize("widths,what", [([1] + [2] * 65 + [200, 50, 10, 80, 3], np.isnan),
                                         ([1] + [2] * 65, np.isinf), ([1] + [2] * 63 + [100, 2], np.isinf)])
def test_counts_that_wrap_to_zero(widths, what):
    """2^64 paths wrap to a count of zero: 1 / 0 is infinite (where the search ends there)
    and 0 x inf NaN from there up.  Each dependency and betweenness must be the same
    number, infinity or NaN as the batched engine's; in lists that a warp sums (80 and 200
    entries) and that a lane does."""
    start = np.concatenate([[0], np.cumsum(widths)])
    u, v = [], []
    for i in range(len(widths) - 1):
        a, b = np.meshgrid(np.arange(start[i], start[i + 1]), np.arange(start[i + 1], start[i + 2]))
        u.append(a.ravel())
        v.append(b.ravel())
    for symmetric in (False, True):
        hg = gu.HostGraph.from_edges(int(start[-1]), np.concatenate(u), np.concatenate(v), symmetric=symmetric)
        g = gu.Graph(hg)
        srcs = np.resize([v for v in (0, 1, 2, 3, 5, 131, 140, 400, hg.n - 1) if v < hg.n], 70).astype(np.int32)
        s = torch.as_tensor(srcs, device="cuda")
        out = []
        for batch in (0, 64):
            bc = torch.empty(hg.n, dtype=torch.float64, device="cuda")
            delta = torch.full((len(srcs), hg.n), -7.0, dtype=torch.float64, device="cuda")
            g.bc(s, bc, delta_dev=delta, batch=batch)
            assert (g.level_profile() == []) == (batch == 0)
            out.append((bc.cpu().numpy(), delta.cpu().numpy()))
        assert symmetric or what(out[1][1]).any()
        for mine, ref in zip(*out):
            np.testing.assert_array_equal(np.isnan(mine), np.isnan(ref))
            np.testing.assert_allclose(mine, ref, rtol=RTOL, atol=0)  # infinities and NaN equal theirs


@pytest.mark.parametrize("n,m,k,small", [(3000, 120000, 16, False), (3000, 120000, 17, True), (3000, 60000, 5, True),
                                         (3000, 180000, 100, False), (3000, 180000, 101, True), (3000, 180000, 401, False),
                                         (5000, 430000, 40, False), (900, 260000, 20, False), (900, 260000, 100, True),
                                         (3000, 450000, 4, True)])
def test_dense_graphs(n, m, k, small):
    """Most lists long: few sources, and many on the largest graphs, go to the batched
    engine, which reads the adjacency once for a pass's sources, unless two levels reach
    everything.  Either engine's counts and betweenness are right."""
    hg = gu.HostGraph.er(n, m, seed=1)
    g = gu.Graph(hg)
    srcs = gu.sources(n, k, seed=2)
    s = torch.as_tensor(srcs, device="cuda")
    sig = torch.empty((k, n), dtype=torch.int64, device="cuda")
    bc = torch.empty(n, dtype=torch.float64, device="cuda")
    g.sigma(s, sig)
    assert (g.level_profile() == []) == small
    np.testing.assert_array_equal(sig.cpu().numpy().view(np.uint64), oracle.sigma_multi(hg.R, hg.C, n, srcs, nthreads=8)[1])
    g.bc(s, bc)
    assert (g.level_profile() == []) == small
    np.testing.assert_allclose(bc.cpu().numpy(), oracle.bc(hg.R, hg.C, n, srcs, nthreads=8), rtol=RTOL, atol=0)


def test_searches_that_reach_everything():
    """The last level is not pushed once all vertices with in-edges, and the source, are
    reached: sources without in-edges, with all others on one level, one vertex short of
    everything, a vertex that only another source reaches, and a single vertex."""
    n = 70
    a, b = np.meshgrid(np.arange(n), np.arange(n))
    check(gu.HostGraph.from_edges(n, a.ravel(), b.ravel()), np.arange(n, dtype=np.int32))  # complete
    below = a.ravel() < b.ravel()
    check(gu.HostGraph.from_edges(n, a.ravel()[below], b.ravel()[below], symmetric=False), np.arange(n, dtype=np.int32), True)
    for extra in ([], [(68, 69)], [(69, 0)], [(0, 69), (69, 68)]):
        u = np.array([0] * 30 + [1 + i % 30 for i in range(200)] + [e[0] for e in extra])
        v = np.array(list(range(1, 31)) + [31 + (7 * i) % 38 for i in range(200)] + [e[1] for e in extra])
        check(gu.HostGraph.from_edges(n, u, v, symmetric=False), np.array([0, 1, 30, 31, 68, 69], np.int32), True)
    check(gu.HostGraph(np.zeros(2, np.int32), np.zeros(0, np.int32), 1), np.array([0], np.int32))
