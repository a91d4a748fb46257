"""Load-balanced search at the edges of its tiles (4096 counts), windows (1024 slots),
pieces (4096 slots) and of the tile sums that every tile adds up itself (4096 tiles):
scan, owners and total exact against numpy, nothing written outside the result."""
import numpy as np
import pytest

import gu

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def check(counts, r_off=0, s_off=0, c_off=0):
    counts = np.asarray(counts, np.int32)
    n, total = len(counts), int(counts.sum(dtype=np.int64))
    cbuf = torch.zeros(n + 4, dtype=torch.int32, device="cuda")
    cbuf[c_off:c_off + n] = torch.as_tensor(counts, device="cuda")
    sbuf = torch.full((n + 8,), -5, dtype=torch.int32, device="cuda")
    rbuf = torch.full((total + 16,), -5, dtype=torch.int32, device="cuda")
    t = gu.lbs(cbuf[c_off:c_off + n], sbuf[s_off:s_off + n], rbuf[r_off:r_off + total])
    assert t == total
    want = np.cumsum(counts, dtype=np.int64) - counts
    np.testing.assert_array_equal(sbuf[s_off:s_off + n].cpu().numpy(), want)
    owners = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.as_tensor(counts, device="cuda").long())
    assert torch.equal(rbuf[r_off:r_off + total].long(), owners)
    assert (rbuf[:r_off] == -5).all() and (rbuf[r_off + total:] == -5).all()
    assert (sbuf[:s_off] == -5).all() and (sbuf[s_off + n:] == -5).all()


@pytest.mark.parametrize("r_off", [0, 1, 2, 3])
@pytest.mark.parametrize("total", [1, 3, 4, 5, 1022, 1023, 1024, 1025, 1027, 2049, 4095, 4096, 4097, 4100, 8193, 100_003])
def test_one_item_and_windows(total, r_off):
    check([total], r_off)
    check([0, 0, total, 0], r_off)
    check([1] * min(total, 255) + [max(0, total - 255)], r_off)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 255, 256, 257, 4095, 4096, 4097, 12_289])
def test_tiles_with_mixed_counts(n):
    rng = np.random.default_rng(n)
    for offs in ((0, 0, 0), (1, 3, 2)):
        check(rng.integers(0, 5, n), *offs)
        heavy = rng.integers(0, 4, n)
        heavy[rng.integers(0, n, max(1, n // 100))] = rng.integers(31, 34)
        heavy[rng.integers(0, n, 2)] = [9000, 5]
        check(heavy, *offs)


@pytest.mark.parametrize("r_off", range(8))
def test_short_lists_searches_and_pieces(r_off):
    """The forms that a warp's slots are written in, at every alignment of the result and
    next to each other: short lists (counts up to 4) with few and with many lanes in a
    bank, items without slots between the others, searches up to 4096 slots, and pieces
    of 2048 beyond, which start and end inside items."""
    rng = np.random.default_rng(r_off)
    for n in (256, 300, 513):
        for c in (1, 2, 3, 4, 5, 8, 15, 16, 17, 40):
            check(np.full(n, c), r_off)
        for p in (0.02, 0.3):  # few items own slots
            check(np.where(rng.random(n) < p, rng.integers(1, 5, n), 0), r_off)
            check(np.where(rng.random(n) < p, rng.integers(1, 90, n), 0), r_off)
    for last in (15, 16, 17, 2047, 2048, 2049, 4111, 6001):  # 4080 slots and the last item's
        check([16] * 255 + [last], r_off)
        check([last] + [16] * 255 + [0, 0, 3], r_off)
    check(np.concatenate([rng.integers(0, 5, 256), rng.integers(0, 40, 256), rng.integers(100, 900, 256), [4] * 256,
                          [0] * 256, [70000], rng.integers(0, 3, 700)]), r_off)


def test_warps_write_more_of_a_large_total():
    """Beyond 4096 slots a warp writes 2^-13 of the total itself: 5500 of 46 M, next to
    warps with more."""
    rng = np.random.default_rng(1)
    counts = np.full(2_100_000, 21)
    counts[rng.integers(0, len(counts), 50)] = 3000
    counts[::7] += 1
    check(counts, 1)


def test_more_tiles_than_are_added_directly():
    rng = np.random.default_rng(2)
    n = 4096 * 4097 + 11
    check(rng.integers(0, 3, n))
    counts = np.zeros(n, np.int32)
    counts[-1] = -1  # the last tile's negative count rejects the call
    c = torch.as_tensor(counts, device="cuda")
    res = torch.full((16,), -7, dtype=torch.int32, device="cuda")
    with pytest.raises(gu.GuError) as e:
        gu.lbs(c, torch.empty_like(c), res)
    assert e.value.status == 1 and (res == -7).all()
