"""Submissions of an insert and a delete batch of unlike sizes: each side takes the
path of its own size (one fused launch up to RG_OPT_FUSED_MAX edges), and the
values are those of two calls."""
import numpy as np
import pytest

import risgraph_b200 as rg
from risgraph_b200 import gen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graphs():
    scale = 14
    V = 1 << scale
    pairs = gen.rmat(scale, n_edges=16 * V, seed=21)
    root = gen.max_out_degree_vertex(pairs, V)
    n = 12 * V
    made = []
    for _ in range(2):
        g = rg.Graph(V, len(pairs), weighted=True)
        g.add_pairs(pairs[:n], want_old=False)
        g.build_tree("sssp", root)
        made.append(g)
    yield made[0], made[1], gen.edges_with_weights(pairs, True), n
    for g in made:
        g.close()


@pytest.mark.parametrize("n_add,n_del", [(1, 2049), (2049, 1), (16, 3000), (3000, 17), (2048, 2049), (2049, 2048),
                                         (2049, 2049), (2048, 2048), (5000, 2500)])
def test_unlike_sides(graphs, n_add, n_del):
    g, h, e, n = graphs
    for adds, dels in ((e[n:n + n_add], e[:n_del]), (e[:n_del][:n_add], e[n:n + n_add][:n_del])):
        g.apply_add_del("sssp", adds, dels)
        h.apply_add("sssp", adds)
        h.apply_del("sssp", dels)
        np.testing.assert_array_equal(g.values(), h.values())
        np.testing.assert_array_equal(g.degrees()[1], h.degrees()[1])


@pytest.mark.parametrize("small_first", [False, True])
def test_the_small_side_is_one_launch(graphs, small_first):
    """A large batch, and one edge beside it that changes no label."""
    g, _, e, n = graphs
    own = np.zeros(1, rg.EDGE_DTYPE)   # a self-loop
    own["src"] = own["dst"] = own["data"] = 5

    def launches(call):
        at = g.launch_count()
        call()
        return g.launch_count() - at

    if small_first:
        g.apply_add("sssp", e[n:n + 3000])
        alone = launches(lambda: g.apply_del("sssp", e[n:n + 3000]))
        g.apply_add("sssp", e[n:n + 3000])
        both = launches(lambda: g.apply_add_del("sssp", own, e[n:n + 3000]))
        g.apply_del("sssp", own)
    else:
        g.apply_add("sssp", own)
        alone = launches(lambda: g.apply_add("sssp", e[n:n + 3000]))
        g.apply_del("sssp", e[n:n + 3000])
        both = launches(lambda: g.apply_add_del("sssp", e[n:n + 3000], own))
        g.apply_del("sssp", e[n:n + 3000])
    assert both == alone + 1
