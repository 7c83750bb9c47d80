"""Aggregating a graph whose edges lie in a few communities takes no scratch in
proportion to them: what a run allocates beside the workspace stays below two
bytes an edge (the uploaded graph and the workspace are about 27)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deterministic", [False, True])
def test_few_large_communities(cuda, deterministic):
    G = cuda.Graph.planted_partition(200000, 50000, 64.0, 0.95, 1)
    G.modularity(np.zeros(G.span, np.uint32))  # (allocates the workspace)
    before = G.device_bytes()
    r = cuda.louvain_static(G, cuda.LouvainOptions(deterministic=deterministic))
    assert r.passes > 1
    assert G.device_bytes() - before <= 2 * G.size
    # the aggregated rows are those of the membership: the totals add up, on every level
    assert r.communityWeight[np.unique(r.membership)].sum() == G.edge_weight()
