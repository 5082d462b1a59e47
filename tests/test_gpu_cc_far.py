"""Connectivity of a graph whose parents are larger than the L2 and whose average
degree is high: the hooking passes are left out. Against the labels by BFS."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("draws", [1 << 27, (1 << 26) + (1 << 25)])  # average degree 16 (left out) and 12 (not)
def test_labels(ctx, draws):
    import byo_gb300 as byo
    G = byo.Graph.generate(ctx, "er", seed=11, n=1 << 24, draws=draws)
    assert (G.M() >= 15 << 24) == (draws == 1 << 27)
    lab = byo.SimpleUnionAsync(G)
    assert np.array_equal(lab, byo.bfs_cc(G))
    G.close()
