"""Triangle counts where rows and lists are short and there are many: rows around
32 neighbours, lists around the 16 entries that half a warp takes, as many
vertices as a launch of their own takes and fewer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [9, 17, 18, 33, 34])
@pytest.mark.parametrize("vertices", [40000, 70000])
def test_many_cliques(ctx, size, vertices):
    """Disjoint cliques (every |N+| from 0 to size - 1), with a bridge between neighbouring ones."""
    import byo_gb300 as byo
    count = vertices // size + 1
    i, j = np.triu_indices(size, 1)
    base = np.arange(count, dtype=np.int64)[:, None] * size
    src = np.concatenate([(base + i).ravel(), base[:-1, 0]])
    dst = np.concatenate([(base + j).ravel(), base[1:, 0] + 1])
    p = np.random.default_rng(size).permutation(count * size)
    src, dst = p[src], p[dst]
    k = np.sort(np.concatenate([src << 32 | dst, dst << 32 | src]))
    off = np.zeros(count * size + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(k >> 32, minlength=count * size))
    G = byo.Graph.from_csr(ctx, off, (k & 0xFFFFFFFF).astype(np.uint32))
    assert byo.Triangle_degree_ordering(G) == count * size * (size - 1) * (size - 2) // 6
    G.close()
