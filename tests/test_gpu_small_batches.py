"""Unsorted batches around the sizes at which the small sort splits (tiles of 32
keys, eighths of the batch, its limit of 4096), with and without equal keys."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _keys(kind, count, n, rng):
    if kind == "equal":
        return np.full(count, ((n - 1) << 32) | 5, np.uint64)
    if kind == "falling":  # distinct
        return ((np.arange(count, dtype=np.uint64)[::-1] << np.uint64(32)) | np.uint64(n - 1))
    high = 40 if kind == "repeated" else n
    return (rng.integers(0, high, count).astype(np.uint64) << np.uint64(32)) | rng.integers(0, high, count).astype(np.uint64)


@pytest.mark.parametrize("container", ["pma", "pcsr", "vos"])
@pytest.mark.parametrize("kind", ["random", "repeated", "equal", "falling"])
@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 255, 257, 1024, 1025, 2047, 2049, 4095, 4096, 4097])
def test_insert_and_remove(ctx, container, kind, count):
    import byo_gb300 as byo
    rng = np.random.default_rng(count)
    n = 8192
    first = np.unique(_keys("random", 20000, n, rng))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount((first >> np.uint64(32)).astype(np.int64), minlength=n))
    G = byo.Graph.from_csr(ctx, off, first.astype(np.uint32), container=container)
    batch = _keys(kind, count, n, rng)
    steps = ((G.insert_batch, np.union1d(first, batch), np.setdiff1d(batch, first).size),
             (G.remove_batch, np.setdiff1d(first, batch), np.unique(batch).size))
    for update, want, changed in steps:
        assert update(batch) == changed
        o, nb = G.export_csr()
        src = np.repeat(np.arange(n, dtype=np.uint64), np.diff(o).astype(np.int64))
        assert np.array_equal((src << np.uint64(32)) | nb, want)
    G.close()
