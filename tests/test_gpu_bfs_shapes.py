"""BFS where the run of small rounds changes path: vertices around the lengths at
which an entry takes a warp or is cut into pieces, hubs around the chunk size of
the round kernels, frontiers around the size that leaves the run, isolated
sources."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, src, dst):
    k = np.unique(np.concatenate([(src << 32) | dst, (dst << 32) | src]))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(k >> 32, minlength=n))
    return off, (k & 0xFFFFFFFF).astype(np.uint32)


def _brooms(lengths):
    """A path whose i-th vertex has lengths[i] leaves, and an isolated vertex at the end."""
    h = len(lengths)
    leaves = h + np.concatenate([[0], np.cumsum(lengths)])
    n = int(leaves[-1]) + 1
    src = np.concatenate([np.arange(h - 1)] + [np.full(k, i) for i, k in enumerate(lengths)])
    dst = np.concatenate([np.arange(1, h), np.arange(h, n - 1)])
    rng = np.random.default_rng(3)
    p = rng.permutation(n)
    return n, p[src].astype(np.int64), p[dst].astype(np.int64), [int(p[0]), int(p[h // 2]), int(p[n - 1]), int(p[h])]


def _fans(width, hubs):
    """A root joined to `hubs` vertices, each joined to the same `width` vertices."""
    n = 1 + hubs + width
    src = np.concatenate([np.zeros(hubs)] + [np.full(width, 1 + i) for i in range(hubs)]).astype(np.int64)
    dst = np.concatenate([np.arange(1, 1 + hubs)] + [np.arange(1 + hubs, n)] * hubs).astype(np.int64)
    return n, src, dst, [0, 1, n - 1]


@pytest.mark.parametrize("graph", [lambda: _brooms([62, 63, 64, 65, 66, 510, 511, 512, 513, 1023, 1024, 1025, 3, 0, 1]),
                                   lambda: _brooms([4093, 4094, 4095, 4096, 4097, 6143, 6144, 6145, 20000]),
                                   lambda: _brooms([65530, 10]), lambda: _brooms([65540, 5, 70000]),
                                   lambda: _fans(700, 93), lambda: _fans(700, 95), lambda: _fans(9000, 40)],
                         ids=["pieces", "chunks", "under_limit", "over_limit", "frontier_under", "frontier_over", "wide"])
def test_bfs_paths(ctx, oracle_mod, graph):
    import byo_gb300 as byo
    from byo_gb300 import _abi
    n, src, dst, sources = graph()
    off, nb = _csr(n, src, dst)
    G = byo.Graph.from_csr(ctx, off, nb)
    for s in sources:
        want = oracle_mod.bfs(off, nb, s)
        for pol in range(6):
            par, lev = byo.BFS(G, s, policy=pol, levels=True)
            assert np.array_equal(par, want[0]) and np.array_equal(lev, want[1]), (s, pol)
    # hubs listed from the round kernels as soon as they have 32 neighbours
    G.set_tuning(hub_min=32)
    for s in sources:
        par, lev = byo.BFS(G, s, policy=_abi.POLICY_BLOCKED, levels=True)
        assert np.array_equal(lev, oracle_mod.bfs(off, nb, s)[1])
        par, lev = byo.BFS(G, s, policy=_abi.POLICY_PUSH, levels=True)
        want = oracle_mod.bfs(off, nb, s)
        assert np.array_equal(par, want[0]) and np.array_equal(lev, want[1])
    G.close()


def test_edge_map_frontier_with_repeats(ctx, oracle_mod):
    """A pushed frontier that holds hubs many times over (more hub chunks than a frontier of distinct vertices has)."""
    import byo_gb300 as byo
    from byo_gb300 import _abi
    n, src, dst, _ = _brooms([5000, 5000, 3])
    off, nb = _csr(n, src, dst)
    G = byo.Graph.from_csr(ctx, off, nb)
    G.set_tuning(hub_min=4096)
    hubs = np.argsort(np.diff(off.astype(np.int64)))[-2:].astype(np.uint32)
    f = byo.BFS_F(G, int(hubs[0]))
    vs = byo.vertexSubset(G, np.tile(hubs, 400))
    out = byo.edgeMap(G, vs, f, flags=64)
    near = np.unique(np.concatenate([nb[off[h]:off[h + 1]] for h in hubs]))
    assert np.array_equal(np.sort(out.to_list()), np.setdiff1d(near, hubs[:1]))
    for o in (out, vs, f):
        o.close()
    G.close()
