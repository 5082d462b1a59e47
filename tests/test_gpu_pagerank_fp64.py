"""PageRank in FP64: sums and shares at the edges of its units (runs of 128
slots, chunks of 512, 8 chunks a vertex), and the shares' quotients, exactly."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n, src, dst):
    k = np.unique(np.concatenate([(src << 32) | dst, (dst << 32) | src]).astype(np.int64))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(k >> 32, minlength=n))
    return off, (k & 0xFFFFFFFF).astype(np.uint32)


def test_shares_are_correctly_rounded(ctx):
    """Stars of 1 to 1000 leaves among 2^19 vertices: the centres' sums are exact,
    so two iterations are known to the last bit."""
    import byo_gb300 as byo
    from byo_gb300 import _abi
    n, most = 1 << 19, 1000
    d = np.arange(1, most + 1)
    centre = np.concatenate([[0], np.cumsum(d + 1)[:-1]])
    leaf = np.concatenate([np.arange(c + 1, c + 1 + k) for c, k in zip(centre, d)])
    off, nb = _csr(n, np.repeat(centre, d), leaf)
    G = byo.Graph.from_csr(ctx, off, nb)
    p = byo.PageRank(G, 0.0, 2, precision=_abi.PR_FP64)
    G.close()
    damping, added = Fraction(0.85), Fraction((1 - 0.85) * (1 / n))
    for c, k in zip(centre.tolist(), d.tolist()):
        first = float(damping * Fraction(k, n) + added)  # one rounding: a fused multiply-add
        share = first / k
        assert p[c + 1] == p[c + k] == float(damping * Fraction(share) + added), k


@pytest.mark.parametrize("degree", [0, 1, 127, 128, 129, 511, 512, 513, 1024, 1025, 4095, 4096, 4097, 4608, 16385])
def test_rows_at_unit_edges(ctx, oracle_mod, degree):
    """33 rows of one length above a sparse rest, with the iterations as one graph
    and launch by launch.  A sum of k terms is off by at most k * 2^-53 of it, on
    either side, and an iteration passes on 0.85 of an error."""
    import byo_gb300 as byo
    from byo_gb300 import _abi
    rng = np.random.default_rng(degree)
    n, rows = 20011, 33
    src, dst = [rng.integers(rows, n, 3 * n)], [rng.integers(rows, n, 3 * n)]
    for r in range(rows):
        src.append(np.full(degree, r))
        dst.append(rows + rng.permutation(n - rows)[:degree])
    src, dst = np.concatenate(src), np.concatenate(dst)
    keep = src != dst
    off, nb = _csr(n, src[keep], dst[keep])
    want, it, _ = oracle_mod.pagerank(off, nb, 0.0, 20)
    G = byo.Graph.from_csr(ctx, off, nb)
    bound = 2 * max(degree, 64) * 2.0 ** -53 / 0.15
    try:
        got = []
        for graphs in (1, 0):
            _abi.check(_abi.lib().byo_ctx_set_pagerank_graphs(ctx.h, graphs))
            p, its, _ = byo.PageRank(G, 0.0, 20, precision=_abi.PR_FP64, info=True)
            assert its == it == 20
            assert np.abs(p / want - 1).max() <= bound
            got.append(p)
        assert np.array_equal(got[0], got[1])
    finally:
        _abi.check(_abi.lib().byo_ctx_set_pagerank_graphs(ctx.h, 1))
        G.close()
