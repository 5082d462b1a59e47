"""Which CSR arrays are taken: every list strictly increasing and below n, at any
place, with lists that start anywhere relative to the four ids a thread reads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 4099


def _csr(seed):
    rng = np.random.default_rng(seed)
    deg = np.where(rng.random(N) < 0.4, 0, rng.integers(1, 9, N))
    deg[7] = 3000  # one long list
    off = np.zeros(N + 1, np.uint64)
    off[1:] = np.cumsum(deg)
    return off, np.concatenate([np.sort(rng.choice(N, d, replace=False)) for d in deg]).astype(np.uint32)


@pytest.mark.parametrize("container", ["csr", "pma", "pcsr", "vos"])
def test_accepted_as_given(ctx, container):
    import byo_gb300 as byo
    off, nb = _csr(1)
    G = byo.Graph.from_csr(ctx, off, nb, container=container)
    o, b = G.export_csr()
    assert np.array_equal(o, off) and np.array_equal(b, nb) and np.array_equal(G.degrees(), np.diff(off))
    G.close()


@pytest.mark.parametrize("fault", ["equal", "falling", "id", "offset", "past_m"])
@pytest.mark.parametrize("where", [0, 1, 2, 3, "long", "last"])
def test_refused(ctx, fault, where):
    import byo_gb300 as byo
    off, nb = _csr(2)
    starts = off[:-1][np.diff(off.astype(np.int64)) >= 2].astype(np.int64)
    if where == "long":
        at = int(off[7]) + 1500
    elif where == "last":
        at = int(starts[-1]) + 1
    else:  # the second id of a list, at each place within a thread's four
        at = int(starts[starts % 4 == where][5]) + 1
    if fault == "equal":
        nb[at] = nb[at - 1]
    elif fault == "falling":
        nb[at - 1], nb[at] = nb[at], nb[at - 1]
    elif fault == "id":
        nb[at] = N
    else:
        v = int(np.searchsorted(off, at, side="right")) - 1
        off[max(v, 1)] = off[-1] + np.uint64(1 << 40) if fault == "past_m" else off[max(v, 1) + 1] + np.uint64(1)
    with pytest.raises(byo.ByoError):
        byo.Graph.from_csr(ctx, off, nb)
