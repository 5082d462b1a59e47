"""byte-PD integers of one to five bytes at every alignment of the decoder's
words and windows, both ways, and integers that it must refuse."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lists(rng, degrees, widths, n):
    """Sorted lists whose differences take the given numbers of bytes, about a
    quarter of them at the ends of their range."""
    nb = []
    for d in degrees:
        w = rng.choice(widths, d)
        lo, hi = 1 << (7 * (w - 1)), (1 << (7 * w)) - 1
        gap = np.where(rng.random(d) < 0.25, np.where(rng.random(d) < 0.5, lo, hi), rng.integers(lo, hi + 1))
        ids = np.cumsum(gap)
        nb.append(ids[ids < n])
    off = np.concatenate([[0], np.cumsum([x.size for x in nb])])
    return off, np.concatenate(nb).astype(np.uint32)


def _both_ways(ctx, O, off, nb, P):
    import byo_gb300 as byo
    bo, dg, data = O.bytepd_encode(off, nb, P)
    G = byo.Graph.from_bytepd(ctx, bo, dg, data, block=P)
    o2, n2 = G.export_csr()
    assert np.array_equal(o2, off) and np.array_equal(n2, nb)
    b2, d2, x2 = G.to_bytepd(P)
    assert np.array_equal(b2, bo) and np.array_equal(d2, dg) and bytes(x2) == bytes(data)
    G.close()


@pytest.mark.parametrize("P", [1, 2, 31, 33, 64, 127, 1000])
@pytest.mark.parametrize("widths", [[1], [2], [3], [1, 2], [1, 2, 3]])
def test_widths(ctx, oracle_mod, widths, P):
    rng = np.random.default_rng(len(widths) * 100 + widths[-1])
    n = 1 << 22
    degrees = np.concatenate([np.arange(0, 300), rng.integers(1, 40, 700), [4000, 0, 1]])
    off, nb = _lists(rng, degrees, widths, n)
    off = np.concatenate([off, np.full(n + 1 - off.size, off[-1])]).astype(np.uint64)
    _both_ways(ctx, oracle_mod, off, nb, P)


def test_wide_ids(ctx, oracle_mod):
    """Differences of four and five bytes: ids from 2^28 up."""
    n = (1 << 28) + (1 << 20)
    rng = np.random.default_rng(5)
    lists = []
    for d in range(1, 60):
        far = (1 << 28) + np.sort(rng.choice(1 << 20, d, replace=False))
        near = np.sort(rng.choice(1 << 21, d, replace=False))
        lists.append(np.concatenate([near, far]))
    off = np.concatenate([[0], np.cumsum([x.size for x in lists])])
    off = np.concatenate([off, np.full(n + 1 - off.size, off[-1])]).astype(np.uint64)
    _both_ways(ctx, oracle_mod, off, np.concatenate(lists).astype(np.uint32), 64)


@pytest.mark.parametrize("at", [0, 1, 2, 3, 29, 30, 31, 122, 123, 124, 125])
@pytest.mark.parametrize("fault", ["zero", "six bytes", "cut"])
def test_refused(ctx, fault, at):
    """130 differences of one byte after the first, one of them replaced at a
    chosen place."""
    import byo_gb300 as byo
    body = np.ones(130, np.uint8)
    if fault == "zero":
        body[at] = 0
    elif fault == "six bytes":
        body[at:at + 5] = 0x80
    else:
        body[at:] |= 0x80
    data = np.concatenate([np.array([131, 0], np.uint32).view(np.uint8), [np.uint8(5)], body]).astype(np.uint8)
    bo = np.array([0] + [data.size] * 400, np.uint64)
    dg = np.array([131] + [0] * 399, np.int32)
    if fault == "six bytes":  # the bytes that went are made up for, so only the long integer is wrong
        data = np.concatenate([data, np.ones(5, np.uint8)])
        bo[1:] = data.size
    with pytest.raises(byo.ByoError) as e:
        byo.Graph.from_bytepd(ctx, bo, dg, data)
    assert e.value.code == byo._abi.BYO_EINVAL
