"""The grid engine (levels and deletion repairs in one persistent launch): every
kind of level it runs, against the oracle, at frontiers on both sides of its
limits, and against the graph-driven loop that served graphs run
(RG_OPT_CLUSTER_EDGES 0)."""
import threading

import numpy as np
import pytest

import risgraph_b200 as rg
from risgraph_b200 import gen

from helpers import ALGOS, WEIGHTED, edges_of, gpu_graph, oracle_graph

pytestmark = pytest.mark.gpu

# builds: by pushes alone (frontiers of a few hundred thousand vertices, several prefix rounds per piece), one-CTA
# levels off, every level a pull or a bottom-up search
MODES = {"push": {"dense_pull": 0, "bfs_bottom_up": 0}, "push_no_tiny": {"dense_pull": 0, "tiny_edges": 0},
         "pull": {"dense_pull": 1, "pull_div": 1 << 30, "bfs_bottom_up": 0}, "default": {}}


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("mode", sorted(MODES))
def test_engine_builds_equal_graph_driven_builds(algo, mode):
    scale = 18
    V = (1 << scale) - 12345
    pairs = gen.rmat(scale, n_edges=8 * V, seed=3) % V
    root = gen.max_out_degree_vertex(pairs, V)
    g = gpu_graph(algo, V, pairs)
    for k, v in MODES[mode].items():
        g.set_option(k, v)
    total = g.build_tree(algo, root)
    val, _, _ = g.labels()
    init = np.arange(V) if algo == "wcc" else np.full(V, {"bfs": 65536, "sssp": 1 << 27, "sswp": 0}[algo])
    assert total >= (val != init.astype(np.uint64)).sum() - 1   # every label that left its init value but the root's
    sizes, scanned = g.level_trace()
    assert sizes[0] == (V if algo == "wcc" else 1) and (sizes > 0).all() and scanned > 0
    assert (g.level_device_times() >= 0).all()
    g.set_option("cluster_edges", 0)   # the same build through the graph-driven loop
    g.build_tree(algo, root)
    np.testing.assert_array_equal(g.values(), val)
    g.close()


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("fanout", [1, 1023, 1024, 1025, 4095, 4097, 200_001])
def test_engine_frontier_limits(algo, fanout):
    """A root with `fanout` children, each with one child of its own: frontiers at the staged limit, levels at the
    one-CTA slot limit, a hub's list over every CTA; then the root's edges go, half at a time."""
    V = 2 * fanout + 2
    kids = np.arange(1, fanout + 1)
    pairs = np.concatenate([np.stack([np.zeros(fanout, int), kids], 1), np.stack([kids, kids + fanout], 1),
                            [[V - 2, V - 1]]]).astype(np.uint64)
    directed = algo != "wcc"
    g = gpu_graph(algo, V, pairs)
    g.set_option("dense_pull", 0)
    g.set_option("bfs_bottom_up", 0)
    g.set_option("fused_max", 0)
    e = edges_of(algo, pairs)
    g.build_tree(algo, 0)
    for lo, hi in ((0, 0), (0, fanout // 2), (fanout // 2, fanout)):
        if hi > lo:
            g.apply_del(algo, e[lo:hi], directed)
        left = pairs[hi:]
        og = oracle_graph(algo, V, left)
        og.build_tree(0)
        val, par, pw = g.labels()
        np.testing.assert_array_equal(val, og.labels()[0])
        assert og.validate(val, par, pw, 0) == 0
    g.apply_add(algo, e[:fanout], directed)
    og = oracle_graph(algo, V, pairs)
    og.build_tree(0)
    np.testing.assert_array_equal(g.values(), og.labels()[0])
    g.close()


def test_engine_level_bound_is_a_status():
    """A chain longer than RG_OPT_MAX_LEVELS ends with RG_ETIMEOUT, and the graph works afterwards."""
    V = 5000
    chain = np.stack([np.arange(V - 1), np.arange(1, V)], 1).astype(np.uint64)
    g = gpu_graph("bfs", V, chain)
    g.set_option("max_levels", 100)
    with pytest.raises(rg.RGError) as err:
        g.build_tree("bfs", 0)
    assert err.value.status == 6
    g.set_option("max_levels", 0)
    g.build_tree("bfs", 0)
    np.testing.assert_array_equal(g.values(), np.arange(V))
    g.close()


def test_engines_of_two_graphs_from_two_threads():
    """Two graphs built and updated at the same time from two host threads, each on its own stream."""
    scale = 15
    V = 1 << scale
    pairs = gen.rmat(scale, seed=5)
    root = gen.max_out_degree_vertex(pairs, V)
    want = {}
    for algo in ("sssp", "bfs"):
        g = gpu_graph(algo, V, pairs)
        g.set_option("cluster_edges", 0)
        g.build_tree(algo, root)
        want[algo] = g.values()
        g.close()
    bad = []

    def work(algo):
        g = gpu_graph(algo, V, pairs)
        e = edges_of(algo, pairs)[:4000]
        for _ in range(30):
            g.build_tree(algo, root)
            g.apply_del(algo, e)
            g.apply_add(algo, e)
            if not np.array_equal(g.values(), want[algo]):
                bad.append(algo)
        g.close()

    threads = [threading.Thread(target=work, args=(a,)) for a in want]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
