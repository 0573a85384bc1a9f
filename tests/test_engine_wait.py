"""The waits of the grid engine: one that gives up is a status (RG_ETIMEOUT), and
nothing of the stopped call is left for the next one."""
import ctypes

import numpy as np
import pytest

import risgraph_b200 as rg
from risgraph_b200 import gen

from helpers import ALGOS, edges_of, gpu_graph

pytestmark = pytest.mark.gpu

ETIMEOUT = 6


def set_polls(g, polls):
    assert rg.lib().rg_test_wait_polls(g._h, ctypes.c_uint64(polls)) == 0


def stops(call):
    """Whether the call gave up (any other error is one)."""
    try:
        call()
    except rg.RGError as err:
        assert err.status == ETIMEOUT
        return True
    return False


@pytest.mark.parametrize("algo", ALGOS)
def test_a_stopped_build_leaves_nothing_behind(algo):
    """Builds that give up early, midway (pull levels included) and late, each with the next root's build after it."""
    scale = 16
    V = 1 << scale
    pairs = gen.rmat(scale, n_edges=32 * V, seed=9)
    roots = [int(r) for r in np.argsort(-np.bincount(pairs[:, 0].astype(int), minlength=V))[[0, 40, 4000]]]
    g = gpu_graph(algo, V, pairs)
    g.set_option("dense_pull", 1)
    g.set_option("bfs_bottom_up", 0)
    want = {}
    for r in roots:
        g.build_tree(algo, r)
        want[r] = g.values()
    stopped = 0
    for k in range(120):
        set_polls(g, 1 + k // 4)
        stopped += stops(lambda: g.build_tree(algo, roots[k % 3]))
        set_polls(g, 0)
        r = roots[(k + 1) % 3]
        g.build_tree(algo, r)
        np.testing.assert_array_equal(g.values(), want[r])
    assert stopped > 0
    g.close()


@pytest.mark.parametrize("algo", ALGOS)
def test_a_stopped_repair_leaves_nothing_behind(algo):
    """Update batches that give up: the edges are in, the labels come back with a build, later batches are right."""
    scale = 14
    V = 1 << scale
    pairs = gen.rmat(scale, n_edges=16 * V, seed=11)
    root, n, batch = gen.max_out_degree_vertex(pairs, V), 12 * V, 4000
    directed = algo != "wcc"
    g, h = gpu_graph(algo, V, pairs[:n], hint=len(pairs)), gpu_graph(algo, V, pairs[:n], hint=len(pairs))
    h.set_option("cluster_edges", 0)
    e = edges_of(algo, pairs)
    for x in (g, h):
        x.build_tree(algo, root)
    stopped = 0
    for k in range(12):
        adds, dels = e[n + k * batch:n + (k + 1) * batch], e[k * batch:(k + 1) * batch]
        for x in (g, h):
            x.add_edges(adds, directed)
        set_polls(g, 1 + k)
        if stops(lambda: g.apply_del(algo, dels, directed)):
            stopped += 1
        set_polls(g, 0)
        h.apply_del(algo, dels, directed)
        for x in (g, h):
            x.build_tree(algo, root)
        np.testing.assert_array_equal(g.values(), h.values())
        np.testing.assert_array_equal(g.degrees()[0], h.degrees()[0])
    assert stopped > 0
    g.close()
    h.close()


def test_a_long_walk_up_the_tree_is_waited_for():
    """The rescue of one vertex walks 20,000 parents, several times the wait limit set here, while the other CTAs wait."""
    hops, V = 20_000, 250_000
    a, b = 1 + np.arange(hops), 1 + hops + np.arange(hops)
    t = 2 * hops + 1
    chains = [np.stack([np.concatenate([[0], c[:-1]]), c], 1) for c in (a, b)]
    pairs = np.concatenate(chains + [[[a[-1], t], [b[-1], t]]]).astype(np.uint64)
    g = rg.Graph(V, len(pairs))
    g.add_pairs(pairs, want_old=False)
    g.set_option("fused_max", 0)   # the repair goes to the grid
    g.build_tree("bfs", 0)
    before, par, _ = g.labels()
    assert before[t] == hops + 1
    e = np.zeros(1, rg.EDGE_DTYPE)
    e["src"], e["dst"] = par[t], t
    set_polls(g, 1 << 12)
    g.apply_del("bfs", e)
    val, now, _ = g.labels()
    np.testing.assert_array_equal(val, before)
    assert now[t] == (b[-1] if par[t] == a[-1] else a[-1])
    assert g.last_stats()["recomputes"] == 0
    g.close()


def test_a_long_list_in_a_bottom_up_level_is_waited_for():
    """A vertex with three million in-edges, none from the frontier: one warp searches them while the grid waits."""
    front, many = 50_000, 3_000_000
    hub = 1 + front
    pairs = np.concatenate([np.stack([np.zeros(front, int), 1 + np.arange(front)], 1),
                            np.stack([hub + 1 + np.arange(many), np.full(many, hub)], 1)]).astype(np.uint64)
    V = hub + 1 + many
    g = rg.Graph(V, len(pairs))
    g.add_pairs(pairs, want_old=False)
    set_polls(g, 1 << 12)
    g.build_tree("bfs", 0)
    val = g.values()
    assert val[0] == 0 and (val[1:hub] == 1).all() and (val[hub:] == 65536).all()
    g.close()
