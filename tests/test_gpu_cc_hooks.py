"""Connectivity on both sides of the rules that choose its hooking passes: vertex
counts around 2^18, graphs that the first sampling round leaves in many trees
(uniform, matchings, permuted paths) and in few (grids, stars)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEAST = 1 << 18  # vertices from which hooking may run


def _csr(n, src, dst):
    keep = src != dst
    src, dst = src[keep].astype(np.int64), dst[keep].astype(np.int64)
    k = np.unique(np.concatenate([(src << 32) | dst, (dst << 32) | src]))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(k >> 32, minlength=n))
    return off, (k & 0xFFFFFFFF).astype(np.uint32)


def _edges(kind, n):
    rng = np.random.default_rng(n)
    if kind == "sparse":
        return rng.integers(0, n, n), rng.integers(0, n, n)
    if kind == "dense":
        return rng.integers(0, n, 6 * n), rng.integers(0, n, 6 * n)
    if kind == "path":
        p = rng.permutation(n)
        return p[:-1], p[1:]
    if kind == "pairs":
        p = rng.permutation(n)[: n // 2 * 2]
        return p[::2], p[1::2]
    if kind == "stars":  # every 1000th vertex a centre
        v = np.arange(n)
        return v, v - v % 1000
    v = np.arange(n - 512)  # grid
    return np.concatenate([v, v]), np.concatenate([v + 512, v + 1])


@pytest.mark.parametrize("kind", ["sparse", "dense", "path", "pairs", "stars", "grid"])
@pytest.mark.parametrize("n", [LEAST - 1, LEAST, LEAST + 33, 3 * LEAST + 1])
def test_labels(ctx, oracle_mod, kind, n):
    import byo_gb300 as byo
    off, nb = _csr(n, *_edges(kind, n))
    want = oracle_mod.cc(off, nb)
    G = byo.Graph.from_csr(ctx, off, nb)
    for _ in range(5):
        assert np.array_equal(byo.SimpleUnionAsync(G), want)
    G.close()
