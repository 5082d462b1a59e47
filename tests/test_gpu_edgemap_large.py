"""One dense edgeMap round of the sums (PR_F, PR_Delta_F) on graphs large enough to
be planned, bit for bit against a sequential scan: skewed ones (planned), uniform
ones (on their own) and ones whose lists are mostly long (planned without a look)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DENSE_ONLY, NO_OUTPUT = 1024, 1
GRAPHS = {"skewed": dict(kind="rmat", lg_n=22, draws=6 << 20), "uniform": dict(kind="er", n=700001, draws=6 << 20),
          "dense": dict(kind="er", n=70001, draws=5 << 19)}


@pytest.mark.parametrize("container", ["csr", "pma", "vos"])
@pytest.mark.parametrize("graph", list(GRAPHS))
def test_one_round(ctx, graph, container):
    import torch

    import byo_gb300 as byo
    G = byo.Graph.generate(ctx, seed=5, container=container, **GRAPHS[graph])
    off, nbr = G.export_csr()
    off, n = off.astype(np.int64), G.N()
    assert G.M() > (1 << 22 if graph == "dense" else 1 << 23) and (G.M() > 56 * n) == (graph == "dense")
    deg = np.diff(off)
    v = np.repeat(np.arange(n), deg)
    rng = np.random.default_rng(9)
    for partial in (False, True):
        x, first = rng.standard_normal(n), np.where(rng.random(n) < 0.3, 0.0, rng.random(n))
        member = rng.random(n) < 0.3 if partial else np.ones(n, bool)
        vs = byo.vertexSubset(G, np.flatnonzero(member).astype(np.uint32)) if partial else byo.vertexSubset.all(G)
        keep = member[nbr]
        reach = np.bincount(v[keep], minlength=n) > 0
        want = first.copy()
        np.add.at(want, v[keep], x[nbr[keep]])  # one after the other
        delta, ngh = (torch.from_numpy(a).cuda() for a in (np.stack([x, x], 1).ravel(), first.copy()))
        torch.cuda.synchronize()
        out = byo.edgeMap(G, vs, byo.PR_Delta_F(G, delta, ngh), flags=DENSE_ONLY)
        assert np.array_equal(ngh.cpu().numpy(), want)
        assert np.array_equal(np.sort(out.to_list()), np.flatnonzero(reach & (first == 0.0)))
        out.close()
        want = first.copy()
        np.add.at(want, v[keep], (x / np.maximum(deg, 1))[nbr[keep]])
        pc, pn = (torch.from_numpy(a.copy()).cuda() for a in (x, first))
        torch.cuda.synchronize()
        out = byo.edgeMap(G, vs, byo.PR_F(G, pc, pn), flags=DENSE_ONLY)
        assert np.array_equal(pn.cpu().numpy(), want)
        assert np.array_equal(np.sort(out.to_list()), np.flatnonzero(reach))
        out.close()
        vs.close()
    G.close()
