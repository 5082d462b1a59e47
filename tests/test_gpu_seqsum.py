"""Dense edgeMap sums (PR_F, PR_Delta_F) bit for bit against a sequential scan,
at run lengths around the kernels' limits and for values that leave the fast
path: ties, wide ranges, zeros, signs, infinities and NaNs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 513, 4095, 4096, 4097, 8191, 8192, 8193, 20000]
DENSE_ONLY, NO_OUTPUT = 1024, 1


def _stars():
    """A star per length; hubs first, then the leaves (degree 1, so a leaf's share is its value)."""
    hubs = len(LENGTHS)
    n = hubs + sum(LENGTHS)
    start = hubs + np.concatenate([[0], np.cumsum(LENGTHS)])
    off = np.zeros(n + 1, np.uint64)
    off[1:hubs + 1] = np.cumsum(LENGTHS)
    off[hubs + 1:] = off[hubs] + np.arange(1, n - hubs + 1, dtype=np.uint64)
    nbr = np.concatenate([np.arange(hubs, n), np.repeat(np.arange(hubs), LENGTHS)]).astype(np.uint32)
    return n, hubs, start, off, nbr


def _values(kind, n, rng):
    if kind == "uniform":
        return rng.random(n)
    if kind == "ties":  # halves of the last place of sums between 1 and 2^15
        return rng.integers(0, 4, n) * 2.0 ** -rng.integers(38, 55, n) + (rng.random(n) < 0.5)
    if kind == "wide":
        return 2.0 ** rng.uniform(-80, 80, n)
    if kind == "tiny":  # subnormal sums
        return rng.integers(0, 3, n) * 5e-324
    if kind == "zeros":
        return np.where(rng.random(n) < 0.99, 0.0, rng.random(n))
    if kind == "signed":
        return rng.standard_normal(n) * 2.0 ** rng.integers(-30, 30, n)
    x = rng.random(n)  # special
    at = rng.integers(0, n, 12)
    x[at[:4]], x[at[4:8]], x[at[8:10]], x[at[10:]] = -0.0, np.inf, -np.inf, np.nan
    return x


@pytest.mark.parametrize("partial", [False, True])
@pytest.mark.parametrize("kind", ["uniform", "ties", "wide", "tiny", "zeros", "signed", "special"])
def test_dense_sums(ctx, kind, partial):
    import torch

    import byo_gb300 as byo
    rng = np.random.default_rng(7)
    n, hubs, start, off, nbr = _stars()
    G = byo.Graph.from_csr(ctx, off, nbr)
    x = _values(kind, n, rng)
    first = np.where(np.arange(n) % 3 == 0, 0.0, rng.random(n))
    member = rng.random(n) < 0.6 if partial else np.ones(n, bool)
    vs = byo.vertexSubset(G, np.flatnonzero(member).astype(np.uint32)) if partial else byo.vertexSubset.all(G)
    want, zero = first.copy(), np.zeros(n, bool)
    for h in range(hubs):
        acc = float(first[h])
        for u in range(start[h], start[h + 1]):
            if member[u]:
                zero[h] |= acc == 0.0
                acc += float(x[u])
        want[h] = acc
    deg = np.diff(off.astype(np.int64))
    with np.errstate(invalid="ignore", over="ignore"):
        for h in range(hubs):  # a leaf's only neighbour is its hub
            if member[h]:
                u = slice(start[h], start[h + 1])
                zero[u] = first[u] == 0.0
    # PR_Delta_F: the values are given, marked where the sum was 0 before an update
    delta = torch.from_numpy(np.stack([x, x], 1).ravel().copy()).cuda()
    ngh = torch.from_numpy(first.copy()).cuda()
    torch.cuda.synchronize()
    out = byo.edgeMap(G, vs, byo.PR_Delta_F(G, delta, ngh), flags=DENSE_ONLY)
    got = ngh.cpu().numpy()
    with np.errstate(invalid="ignore", over="ignore"):
        for h in range(hubs):
            if member[h]:
                u = slice(start[h], start[h + 1])
                want[u] = first[u] + x[h]
    assert np.array_equal(got, want, equal_nan=True)
    assert np.array_equal(np.sort(out.to_list()), np.flatnonzero(zero))
    out.close()
    # PR_F: the values are shares of the source's degree
    pc, pn = torch.from_numpy(x.copy()).cuda(), torch.from_numpy(first.copy()).cuda()
    torch.cuda.synchronize()
    byo.edgeMap(G, vs, byo.PR_F(G, pc, pn), flags=DENSE_ONLY | NO_OUTPUT)
    with np.errstate(invalid="ignore", over="ignore"):
        for h in range(hubs):
            if member[h]:
                u = slice(start[h], start[h + 1])
                want[u] = first[u] + x[h] / deg[h]
    assert np.array_equal(pn.cpu().numpy(), want, equal_nan=True)
    vs.close()
