"""Per-source rows of sigma, distance and delta at the edges of the write-out's tiles
(64 vertices x 64 sources, 8 staged levels): integers exact, delta within 1e-12
relative of the FP64 oracle, nothing written beyond a row's n values."""
import numpy as np
import pytest

import gu
import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def graph(n, kind):
    if kind == "path":  # n levels: most beyond the staged ones
        return gu.HostGraph.from_edges(n, np.arange(n - 1), np.arange(1, n))
    rng = np.random.default_rng(n)
    return gu.HostGraph.from_edges(n, rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n))


@pytest.mark.parametrize("n,k,kind", [(1, 1, "random"), (63, 63, "random"), (64, 64, "random"), (65, 65, "random"),
                                      (130, 129, "random"), (700, 300, "random"), (40, 40, "path"), (200, 70, "path")])
def test_rows_at_tile_edges(n, k, kind):
    hg = graph(n, kind) if n > 1 else gu.HostGraph(np.zeros(2, np.int32), np.zeros(0, np.int32), 1)
    g = gu.Graph(hg)
    srcs = np.arange(k, dtype=np.int32) % n
    ld = n + 3
    s = torch.as_tensor(srcs, device="cuda")
    sig = torch.full((k, ld), -7, dtype=torch.int64, device="cuda")
    d = torch.full((k, ld), -7, dtype=torch.int32, device="cuda")
    g.sigma(s, sig, dist_dev=d, ld=ld)
    rd, rs = oracle.sigma_multi(hg.R, hg.C, n, srcs, nthreads=4)
    np.testing.assert_array_equal(d.cpu().numpy()[:, :n], rd)
    np.testing.assert_array_equal(sig.cpu().numpy().view(np.uint64)[:, :n], rs)
    assert (sig[:, n:] == -7).all() and (d[:, n:] == -7).all()
    only = torch.full((k, ld), -7, dtype=torch.int64, device="cuda")
    g.sigma(s, only, ld=ld)  # without distances
    assert torch.equal(only, sig)
    bc = torch.empty(n, dtype=torch.float64, device="cuda")
    delta = torch.full((k, ld), -7.0, dtype=torch.float64, device="cuda")
    g.bc(s, bc, delta_dev=delta, ld=ld)
    got = delta.cpu().numpy()
    assert (got[:, n:] == -7.0).all()
    for i in range(k):
        _, _, ref = oracle.brandes(hg.R, hg.C, n, int(srcs[i]), "f64")
        np.testing.assert_allclose(got[i, :n], ref, rtol=1e-12, atol=0)
