"""The division on the integer units and the integer sum over a batch's sources, on path
counts of every size: powers of two, counts that need rounding to 53 bits, and counts
that wrapped.  Dependencies within 1e-12 relative of the oracle (60 levels of four
roundings each are below 3e-14)."""
import os

import numpy as np
import pytest

import gu
import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
RTOL = 1e-12


def layers(widths):
    """Complete bipartite layers: the count at a vertex is the product of the widths before."""
    start = np.concatenate([[0], np.cumsum(widths)])
    u, v = [], []
    for i in range(len(widths) - 1):
        a, b = np.meshgrid(np.arange(start[i], start[i + 1]), np.arange(start[i + 1], start[i + 2]))
        u.append(a.ravel())
        v.append(b.ravel())
    return gu.HostGraph.from_edges(int(start[-1]), np.concatenate(u), np.concatenate(v), symmetric=False)


def run(hg, srcs, words):
    os.environ["GU_BC_WORDS"] = words
    if not words:
        del os.environ["GU_BC_WORDS"]
    try:
        s = torch.as_tensor(np.asarray(srcs, np.int32), device="cuda")
        bc = torch.empty(hg.n, dtype=torch.float64, device="cuda")
        delta = torch.full((len(srcs), hg.n), -7.0, dtype=torch.float64, device="cuda")
        gu.Graph(hg).bc(s, bc, delta_dev=delta)
        return bc.cpu().numpy(), delta.cpu().numpy()
    finally:
        os.environ.pop("GU_BC_WORDS", None)


@pytest.mark.parametrize("words", ["", "1", "2", "4"])
@pytest.mark.parametrize("widths", [[2] * 63, [1, 3] * 39, [3] * 39 + [1], [5, 3, 7] * 8, [1, 63, 61, 59, 57, 55, 53, 51, 47, 43]])
def test_counts_of_every_size(widths, words):
    hg = layers(widths)
    srcs = np.arange(min(hg.n, 150), dtype=np.int32)
    bc, delta = run(hg, srcs, words)
    for i in range(0, len(srcs), 7):
        _, _, ref = oracle.brandes(hg.R, hg.C, hg.n, int(srcs[i]), "pull")
        np.testing.assert_allclose(delta[i], ref, rtol=RTOL, atol=0)
    np.testing.assert_allclose(bc, oracle.bc(hg.R, hg.C, hg.n, srcs, pull=True, nthreads=8), rtol=RTOL, atol=0)


@pytest.mark.parametrize("k", [1, 64, 65, 200, 1024])
def test_sum_over_sources(k):
    """Terms of very different sizes, zeros and sources at the vertex itself."""
    rng = np.random.default_rng(k)
    n = 9000
    u = np.concatenate([np.zeros(4000, np.int64), rng.integers(0, n, 30000)])
    v = np.concatenate([np.arange(1, 4001), rng.integers(0, n, 30000)])
    hg = gu.HostGraph.from_edges(n, u, v)
    srcs = gu.sources(n, k, seed=1)
    ref = oracle.bc(hg.R, hg.C, n, srcs, nthreads=8)
    g = gu.Graph(hg)
    s = torch.as_tensor(srcs, device="cuda")
    for batch in (64, 1024):
        bc = torch.empty(n, dtype=torch.float64, device="cuda")
        g.bc(s, bc, batch=batch)
        np.testing.assert_allclose(bc.cpu().numpy(), ref, rtol=RTOL, atol=0)
