"""Work that a launch of the grid engine leaves to another: push levels to the
graph-driven loop, and repairs on half the SMs, at a level or in the invalidation,
to a launch on all.  From builds and repairs, at frontiers in either queue, and
from the insert batch of a submission whose delete batch waits for it."""
import ctypes

import numpy as np
import pytest

import risgraph_b200 as rg
from risgraph_b200 import gen

from helpers import ALGOS, WEIGHTED, edges_of

pytestmark = pytest.mark.gpu

SCALE = 15
# (a level is measured by its slots only when its frontier is too large to be staged whole: 2,048 vertices)
SLOTS = [1, 60_000, 300_000, 1 << 40]


# vertices of a frontier or a reset set
VERTICES = [1, 700, 6000]


def set_slots(g, n):
    assert rg.lib().rg_test_push_slots(g._h, ctypes.c_uint64(n)) == 0


def set_vertices(g, n):
    assert rg.lib().rg_test_half_vertices(g._h, ctypes.c_uint64(n)) == 0


def bridged(algo):
    """An RMAT graph and, apart, the root: the edge between them brings the whole graph to it or takes it away."""
    V0 = 1 << SCALE
    pairs = gen.rmat(SCALE, n_edges=16 * V0, seed=13) + np.uint64(1)
    hub = gen.max_out_degree_vertex(pairs, V0 + 1)
    return V0 + 1, pairs, np.array([[0, hub]], np.uint64)


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("slots", SLOTS)
def test_push_levels_left_to_the_loop(algo, slots):
    compare(algo, lambda g: set_slots(g, slots))


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("vertices", VERTICES)
@pytest.mark.parametrize("slots", [0, 100_000])
def test_repairs_left_to_all_sms(algo, vertices, slots):
    def setup(g):
        set_vertices(g, vertices)
        set_slots(g, slots)

    compare(algo, setup)


def compare(algo, setup):
    """Updates and builds on a graph with `setup` and on one that runs the loop alone."""
    V, pairs, bridge = bridged(algo)
    directed = algo != "wcc"
    g, h = (rg.Graph(V, len(pairs) + 4096, symmetric=not directed, weighted=WEIGHTED[algo]) for _ in range(2))
    h.set_option("cluster_edges", 0)
    setup(g)
    e, b = edges_of(algo, pairs), edges_of(algo, bridge)
    for x in (g, h):
        x.add_pairs(pairs, directed, want_old=False)
        x.build_tree(algo, 0)

    def same():
        val, par, _ = g.labels()
        np.testing.assert_array_equal(val, h.values())
        assert ((par < V) | (par == V)).all()
        sizes, _ = g.level_trace()
        assert (sizes > 0).all()

    same()
    for x in (g, h):      # one edge: what outgrows the one-CTA repair
        x.apply_add(algo, b, directed)
    same()
    for x in (g, h):      # builds, pushes only and as they come
        x.set_option("dense_pull", 0)
        x.set_option("bfs_bottom_up", 0)
        x.build_tree(algo, 0)
    same()
    for x in (g, h):
        x.set_option("dense_pull", 2)
        x.set_option("bfs_bottom_up", 1)
        x.build_tree(algo, 0)
        x.apply_del(algo, b, directed)
    same()
    for x in (g, h):      # the insert's levels are left while the delete batch waits: inline, staged, large
        x.apply_add_del(algo, b, e[:1], directed)
        x.apply_add_del(algo, e[:1], b, directed)
    same()
    for x in (g, h):
        x.apply_add_del(algo, np.concatenate([b, e[:40]]), e[40:90], directed)
    same()
    for x in (g, h):
        x.apply_add_del(algo, e[40:90], np.concatenate([b, e[:40]]), directed)
        x.apply_add_del(algo, np.concatenate([b, e[:3000]]), e[3000:6000], directed)
    same()
    for x in (g, h):      # many tree edges at once, and back
        _, par, pw = x.labels()
        kids = np.nonzero(par < V)[0][::7][:6000]
        d = np.zeros(len(kids), rg.EDGE_DTYPE)
        d["src"], d["dst"], d["data"] = par[kids], kids, pw[kids] if WEIGHTED[algo] else 0
        x.apply_del(algo, d, directed)
        x.apply_add(algo, d, directed)
    same()
    np.testing.assert_array_equal(g.degrees()[0], h.degrees()[0])
    for x in (g, h):
        x.close()
