"""The scan behind plans and compactions at its splits: one tile of 4096 items,
two, and 1024 tiles and more, through the byte offsets of an encoded path."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 4096


@pytest.mark.parametrize("n", [2, 255, TILE - 1, TILE, TILE + 1, 2 * TILE, 2 * TILE + 1, 1023 * TILE + 7, 1024 * TILE,
                               1024 * TILE + 1])
def test_prefixes(ctx, oracle_mod, n):
    import byo_gb300 as byo
    v = np.arange(n, dtype=np.int64)
    nb = np.empty(2 * n - 2, np.uint32)
    nb[0::2], nb[1::2] = v[1:], v[:-1]  # 1 | 0 2 | 1 3 | ... : each vertex's neighbours in turn
    off = np.concatenate([[0], 2 * v[1:] - 1, [2 * n - 2]]).astype(np.uint64)
    G = byo.Graph.from_csr(ctx, off, nb)
    bo, dg, data = G.to_bytepd(64)
    obo, odg, odata = oracle_mod.bytepd_encode(off, nb, 64)
    assert np.array_equal(bo, obo) and np.array_equal(dg, odg) and bytes(data) == bytes(odata)
    G.close()
