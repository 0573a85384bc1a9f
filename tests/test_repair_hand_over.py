"""A deletion repair that the one-CTA levels hand over to the grid: the levels that
they ran count towards the rule that gives up and builds from scratch (only a
repair's first eleven levels may, core/graph.hpp:1252)."""
import numpy as np
import pytest

import risgraph_b200 as rg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster_edges", [0, 65536])
@pytest.mark.parametrize("hops,recomputes", [(5, 1), (14, 0)])
def test_levels_before_the_hand_over_count(cluster_edges, hops, recomputes):
    """A chain of `hops` from the root to a vertex with 1,500 children, more than one CTA takes; its first edge goes."""
    kids = 1500
    chain = np.stack([np.arange(hops), np.arange(1, hops + 1)], 1)
    fan = np.stack([np.full(kids, hops), hops + 1 + np.arange(kids)], 1)
    pairs = np.concatenate([chain, fan]).astype(np.uint64)
    V = hops + 1 + kids
    g = rg.Graph(V, len(pairs))
    g.add_pairs(pairs, want_old=False)
    g.set_option("recompute_min", 1000)
    g.set_option("cluster_edges", cluster_edges)
    g.build_tree("bfs", 0)
    first = np.zeros(1, rg.EDGE_DTYPE)
    first["dst"] = 1
    g.apply_del("bfs", first)
    assert g.last_stats()["recomputes"] == recomputes
    val = g.values()
    assert val[0] == 0 and (val[1:] == 65536).all()
    g.close()
