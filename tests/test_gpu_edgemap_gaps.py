"""One dense edgeMap round of the sums (PR_F, PR_Delta_F), bit for bit against a
sequential scan, on views with and without gaps: lists around the lengths at
which a lane, a warp or a CTA takes them, short ones across a leaf's gap, small
views (shares divided one an edge) and large ones (one a vertex)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DENSE_ONLY, NO_OUTPUT = 1024, 1


def _graph(lengths, rest):
    """A star per length, and `rest` vertices in a ring of degree 4 whose lists cross the leaves of a packed array."""
    hubs = len(lengths)
    first = hubs + np.concatenate([[0], np.cumsum(lengths)])
    src = np.repeat(np.arange(hubs), lengths)
    dst = np.arange(hubs, first[-1])
    r = np.arange(rest)
    src = np.concatenate([src, first[-1] + r, first[-1] + r])
    dst = np.concatenate([dst, first[-1] + (r + 1) % rest, first[-1] + (r + 7) % rest])
    n = int(first[-1]) + rest
    k = np.unique(np.concatenate([src << 32 | dst, dst << 32 | src]))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(np.bincount(k >> 32, minlength=n))
    return n, off, (k & 0xFFFFFFFF).astype(np.uint32)


def _scan(off, nbr, member, x, first):
    want, zero = first.copy(), np.zeros(len(first), bool)
    for v in range(len(first)):
        acc = float(first[v])
        for u in nbr[off[v]:off[v + 1]]:
            if member[u]:
                zero[v] |= acc == 0.0
                acc += float(x[u])
        want[v] = acc
    return want, zero


@pytest.mark.parametrize("partial", [False, True])
@pytest.mark.parametrize("lengths, rest", [([7, 8, 9, 63, 64, 65, 128, 129, 511, 512, 513], 5000),
                                           ([1, 65, 3000, 4095, 4096, 4097, 9000], 30000)], ids=["small", "large"])
@pytest.mark.parametrize("container", ["csr", "pma", "pcsr", "vos"])
def test_one_round(ctx, container, lengths, rest, partial):
    import torch

    import byo_gb300 as byo
    rng = np.random.default_rng(len(lengths) + partial)
    n, off, nbr = _graph(np.array(lengths), rest)
    assert (2 * len(nbr) < 1 << 16) == (rest == 5000) and (len(nbr) > 1 << 16) == (rest == 30000)
    G = byo.Graph.from_csr(ctx, off, nbr, container=container)
    x, first = rng.standard_normal(n), np.where(rng.random(n) < 0.3, 0.0, rng.random(n))
    member = rng.random(n) < 0.3 if partial else np.ones(n, bool)
    vs = byo.vertexSubset(G, np.flatnonzero(member).astype(np.uint32)) if partial else byo.vertexSubset.all(G)
    deg = np.diff(off.astype(np.int64))
    want, zero = _scan(off, nbr, member, x, first)
    delta, ngh = (torch.from_numpy(a).cuda() for a in (np.stack([x, x], 1).ravel(), first.copy()))
    torch.cuda.synchronize()
    out = byo.edgeMap(G, vs, byo.PR_Delta_F(G, delta, ngh), flags=DENSE_ONLY)
    assert np.array_equal(ngh.cpu().numpy(), want)
    assert np.array_equal(np.sort(out.to_list()), np.flatnonzero(zero))
    out.close()
    want, _ = _scan(off, nbr, member, x / np.maximum(deg, 1), first)
    pc, pn = (torch.from_numpy(a.copy()).cuda() for a in (x, first))
    torch.cuda.synchronize()
    byo.edgeMap(G, vs, byo.PR_F(G, pc, pn), flags=DENSE_ONLY | NO_OUTPUT).close()
    assert np.array_equal(pn.cpu().numpy(), want)
    reach = np.array([member[nbr[off[v]:off[v + 1]]].any() for v in range(n)])
    out = byo.edgeMap(G, vs, byo.PR_F(G, pc, pn), flags=DENSE_ONLY)
    assert np.array_equal(np.sort(out.to_list()), np.flatnonzero(reach))
    out.close()
    vs.close()
    G.close()
