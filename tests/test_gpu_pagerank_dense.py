"""PageRank into host arrays on graphs so dense that its workspaces are longer than
the vertices: every vertex heavy (more than 128 neighbours), up to three chunks
of partial sums each, on the first call of a fresh graph and again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dense(n, share):
    rng = np.random.default_rng(n)
    a = np.triu(rng.random((n, n)) < share, 1)
    return a | a.T


def _exact(a, iters):
    n = len(a)
    deg = a.sum(1).astype(np.float64)
    p = np.full(n, 1 / n)
    for _ in range(iters):
        p = 0.85 * (a.astype(np.float64) @ (p / deg)) + 0.15 / n
    return p


# relative error of a vertex: 20 iterations of damped sums (1 / 0.15 of one's error) of at most 1500 terms in
# FP64 (1500 * 2^-53), of 25 FP32 roundings in a row (a lane's 16, the tree, the share) or of 4 compensated
@pytest.mark.parametrize("precision, bound", [("PR_FP32_KAHAN", 2e-6), ("PR_FP64", 2e-12), ("PR_FP32", 1e-5)])
@pytest.mark.parametrize("n, share", [(600, 0.4), (1500, 1.0), (1500, 0.5), (300, 0.9)])
@pytest.mark.parametrize("container", ["csr", "pma"])
def test_dense(ctx, container, n, share, precision, bound):
    import byo_gb300 as byo
    from byo_gb300 import _abi
    a = _dense(n, share)
    off = np.concatenate([[0], np.cumsum(a.sum(1))]).astype(np.uint64)
    G = byo.Graph.from_csr(ctx, off, np.nonzero(a)[1].astype(np.uint32), container=container)
    want = _exact(a, 20)
    first = byo.PageRank(G, eps=0.0, max_iters=20, precision=getattr(_abi, precision))
    assert np.abs(first - want).max() <= bound * want.max()
    assert np.array_equal(byo.PageRank(G, eps=0.0, max_iters=20, precision=getattr(_abi, precision)), first)
    G.close()
