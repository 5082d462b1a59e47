"""Connectivity where its rounds can go wrong: vertex counts at the edges of warps
and around the size from which hooking passes may run, chains as long as the
graph, trees that join in the order of their ids, average degrees on both sides
of the passes' rule, and graphs with a hub of about the share that rules them out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEAST = 1 << 15  # vertices from which hooking may run


def _csr(n, src, dst):
    keep = src != dst
    src, dst = src[keep].astype(np.int64), dst[keep].astype(np.int64)
    k = np.unique(np.concatenate([(src << 32) | dst, (dst << 32) | src]))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(k >> 32, minlength=n))
    return off, (k & 0xFFFFFFFF).astype(np.uint32)


def _edges(kind, n, rng):
    v = np.arange(n - 1)
    if kind == "path":
        return v, v + 1
    if kind == "ladder":  # trees of 8, each joined to the next by its last vertex's second edge
        return np.concatenate([v - v % 8, v]), np.concatenate([v, np.minimum(v + 8, n - 1)])
    if kind == "columns":  # a grid 7 wide, numbered by rows
        return np.concatenate([v, v]), np.concatenate([np.minimum(v + 7, n - 1), np.where(v % 7 < 6, v + 1, v)])
    if kind == "hub":  # the hub takes about a fifth of the vertices, the rest is sparse
        leaves = rng.permutation(n)[: n // 5]
        u, w = rng.integers(0, n, n), rng.integers(0, n, n)
        return np.concatenate([np.full(leaves.size, leaves[0] if leaves.size else 0), u]), np.concatenate([leaves, w])
    per = {"thin": 0.75, "even": 0.8, "thick": 0.9}[kind]  # edges a vertex: average degrees 1.5, 1.6, 1.8
    return rng.integers(0, n, int(per * n)), rng.integers(0, n, int(per * n))


@pytest.mark.parametrize("container", ["csr", "pma"])
@pytest.mark.parametrize("kind", ["path", "ladder", "columns", "hub", "thin", "even", "thick"])
@pytest.mark.parametrize("n", [1, 2, 33, 1025, LEAST - 1, LEAST, 5 * LEAST + 3])
def test_labels(ctx, oracle_mod, container, kind, n):
    import byo_gb300 as byo
    off, nb = _csr(n, *_edges(kind, n, np.random.default_rng(n)))
    G = byo.Graph.from_csr(ctx, off, nb, container=container)
    want = oracle_mod.cc(off, nb)
    for _ in range(3):
        assert np.array_equal(byo.SimpleUnionAsync(G), want)
    G.close()
