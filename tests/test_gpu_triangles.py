"""Triangle counts where the counting kernels change path: rows longer than a
warp's stage, out-lists too long to sort, ranks beyond the bitmaps with short
(hash set) and long (windowed bitmap) out-lists, degree-1 fringes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, src, dst):
    k = np.sort(np.concatenate([(src << 32) | dst, (dst << 32) | src]))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(k >> 32, minlength=n))
    return off, (k & 0xFFFFFFFF).astype(np.uint32)


def _cliques(count, size):
    """`count` disjoint cliques: every |N+| from 0 to size - 1 at every rank."""
    i, j = np.triu_indices(size, 1)
    base = np.arange(count, dtype=np.int64)[:, None] * size
    return count * size, (base + i).ravel(), (base + j).ravel(), count * size * (size - 1) * (size - 2) // 6


def _book(n, spine):
    """Vertices 0..spine-1 in a clique, all joined to every other vertex: rows of n - 1 neighbours."""
    i, j = np.triu_indices(spine, 1)
    k = np.arange(spine, n, dtype=np.int64)
    src = np.concatenate([i] + [np.full(len(k), s) for s in range(spine)])
    dst = np.concatenate([j] + [k] * spine)
    return n, src, dst, spine * (spine - 1) * (spine - 2) // 6 + (n - spine) * spine * (spine - 1) // 2


def _fringe():
    """A triangle, a path of three and a star: only the triangle counts."""
    src = np.array([0, 0, 1, 3, 4] + [10] * 40, np.int64)
    dst = np.array([1, 2, 2, 4, 5] + list(range(11, 51)), np.int64)
    return 64, src, dst, 1


@pytest.mark.parametrize("stage", [0, 513])
@pytest.mark.parametrize("graph", [_fringe, lambda: _book(5000, 2), lambda: _book(1024 + 33, 32), lambda: _cliques(3, 1500),
                                   lambda: _cliques(37, 33), lambda: _cliques(372, 360)],
                         ids=["fringe", "book2", "book32", "cliques1500", "cliques33", "cliques_past_bitmaps"])
def test_triangle_counts(ctx, graph, stage):
    import byo_gb300 as byo
    n, src, dst, want = graph()
    off, nb = _csr(n, src.astype(np.int64), dst.astype(np.int64))
    G = byo.Graph.from_csr(ctx, off, nb)
    G.set_tuning(tc_stage=stage)
    assert byo.Triangle_degree_ordering(G) == want
    G.close()
