"""64-source BFS at the sizes where its kernels change path: vertex counts that do
and do not allow 16-byte level stores, source counts that are no multiple of 8,
runs around the first 32 and the following 128 neighbours of a step, hub chunks
that end inside one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, src, dst):
    k = np.unique(np.concatenate([(src << 32) | dst, (dst << 32) | src]))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(k >> 32, minlength=n))
    return off, (k & 0xFFFFFFFF).astype(np.uint32)


def _graph(n):
    """Hubs of chosen degrees over a sparse random graph, ids permuted."""
    rng = np.random.default_rng(n)
    src, dst = [rng.integers(0, n, n)], [rng.integers(0, n, n)]
    for i, d in enumerate([7, 8, 9, 31, 32, 33, 47, 48, 49, 159, 160, 161, 288, 1023, 1024, 1025, 2500]):
        src.append(np.full(d, i))
        dst.append(rng.choice(n, d, replace=False))
    src, dst = np.concatenate(src).astype(np.int64), np.concatenate(dst).astype(np.int64)
    keep = src != dst
    p = rng.permutation(n)
    return _csr(n, p[src[keep]], p[dst[keep]])


@pytest.mark.parametrize("tuning", [{}, dict(ms_heavy_deg=1, ms_hub_deg=33, ms_push_div=1000000),
                                    dict(ms_heavy_deg=8, ms_hub_deg=161, ms_push_div=1)])
@pytest.mark.parametrize("n,k", [(4096, 64), (4097, 64), (4098, 1), (5003, 63), (4100, 9)])
def test_levels(ctx, oracle_mod, n, k, tuning):
    import byo_gb300 as byo
    off, nb = _graph(n)
    G = byo.Graph.from_csr(ctx, off, nb)
    G.set_tuning(**tuning)
    srcs = np.random.default_rng(k).integers(0, n, k).astype(np.uint32)
    got = byo.BFS_multi(G, srcs)
    for j, s in enumerate(srcs):
        assert np.array_equal(got[j], oracle_mod.bfs(off, nb, int(s))[1]), (j, s)
    G.close()
