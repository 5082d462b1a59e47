"""Triangle counts of graphs whose edges are not all stored at both ends (keys that
were not symmetrised): every u -> v to a higher (degree, id) with the common
ones of both, as the oracle counts them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, arcs):
    k = np.unique(arcs)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(k >> 32, minlength=n))
    return off, (k & 0xFFFFFFFF).astype(np.uint32)


def _random(n, count, seed=1):
    rng = np.random.default_rng(seed)
    arcs = (rng.integers(0, n, count) << 32) | (rng.random(count) ** 2 * n).astype(np.int64)
    return n, arcs[arcs >> 32 != arcs & 0xFFFFFFFF]


def _both(arcs):
    return np.unique(np.concatenate([arcs, (arcs & 0xFFFFFFFF) << 32 | arcs >> 32]))


def _ranked(n, arcs):
    """The arcs, those to a higher (degree, id) and the others."""
    deg = np.bincount(arcs >> 32, minlength=n)
    u, v = arcs >> 32, arcs & 0xFFFFFFFF
    up = (deg[v] << 32 | v) > (deg[u] << 32 | u)
    return arcs[up], arcs[~up]


def _one_less(way):
    """A symmetric graph short of one arc, to the higher or to the lower end."""
    n, arcs = _random(1500, 20000, 2)
    arcs = _both(arcs)
    return n, arcs[arcs != _ranked(n, arcs)[way][7777]]


def _swapped():
    """As many arcs up as down, but not the same: one of each is gone."""
    n, arcs = _random(1500, 20000, 2)
    arcs = _both(arcs)
    up, down = _ranked(n, arcs)
    for i in range(100, 120):
        less = arcs[(arcs != up[i]) & (arcs != down[-i])]
        up2, down2 = _ranked(n, less)
        if len(up2) == len(down2):
            return n, less
    raise AssertionError("no such pair")


def _tournament():
    """Every pair of 700 joined one way: out-lists of up to 700 entries, half of their arcs to higher ranks."""
    i, j = np.triu_indices(700, 1)
    flip = np.random.default_rng(3).random(len(i)) < 0.5
    return 700, np.where(flip, i << 32 | j, j << 32 | i)


def _sinks():
    """9000 vertices with arcs to three hubs, which have arcs to half of them."""
    n, arcs = _random(9003, 60000, 4)
    hubs = np.arange(9000, 9003, dtype=np.int64)
    v = np.arange(9000, dtype=np.int64)
    to = [v << 32 | h for h in hubs]
    back = [h << 32 | v[i % 2::2] for i, h in enumerate(hubs)]
    return n, np.concatenate([arcs, hubs << 32 | np.roll(hubs, 1)] + to + back)


@pytest.mark.parametrize("container", ["csr", "pma"])
@pytest.mark.parametrize("stage", [0, 513])
@pytest.mark.parametrize("graph", [lambda: _random(2000, 60000), lambda: _one_less(0), lambda: _one_less(1), _swapped,
                                   _tournament, _sinks],
                         ids=["random", "up_missing", "down_missing", "swapped", "tournament", "sinks"])
def test_directed_counts(ctx, oracle_mod, graph, stage, container):
    import byo_gb300 as byo
    n, arcs = graph()
    off, nb = _csr(n, arcs)
    G = byo.Graph.from_csr(ctx, off, nb, container=container)
    G.set_tuning(tc_stage=stage)
    want = oracle_mod.triangle_count(off, nb)
    assert byo.Triangle_degree_ordering(G) == want
    G.close()
