"""The kernels of the graph-driven level loop, which served graphs run
(RG_OPT_CLUSTER_EDGES 0) and profile mode steps from the host, where the grid
engine would otherwise take the call: pull levels in one launch, split and in
groups over rows of every kind, cluster levels, and the deletion repair's kernels
for heavy vertices."""
import numpy as np
import pytest

import risgraph_b200 as rg
from oracle import oracle as O
from risgraph_b200 import gen

from helpers import ALGOS, WEIGHTED, edges_of, gpu_graph, oracle_graph
from test_pull_rows import row_graph

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rows():
    """The row graph with its weights and without, and an oracle build of each as loaded and after the re-insertion."""
    V, edges, dels = row_graph(5)
    plain, plain_dels = edges.copy(), dels.copy()
    plain["data"] = plain_dels["data"] = 0
    want = {}

    def values(algo, weighted_copy):
        if (algo, weighted_copy) not in want:
            og = O.OracleGraph(algo, V, len(edges))
            w = WEIGHTED[algo]
            for e in edges:
                og.add_edge(int(e["src"]), int(e["dst"]), int(e["data"]) if w else 0)
            for e in dels:
                og.del_edge(int(e["src"]), int(e["dst"]), int(e["data"]) if w else 0)
            og.build_tree(0)
            first = og.labels()[0].copy()
            for e in dels:
                og.add_edge(int(e["src"]), int(e["dst"]), int(e["data"]) if w else 0)
            og.build_tree(0)
            want[algo, weighted_copy] = first, og.labels()[0].copy()
        return want[algo, weighted_copy]

    return V, {True: (edges, dels), False: (plain, plain_dels)}, values


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("weighted_copy", [False, True])
@pytest.mark.parametrize("split,groups", [(0, 2), (1, 2), (1, 3), (1, 4), (1, 16)])
def test_pull_levels_of_the_loop(rows, algo, weighted_copy, split, groups):
    if WEIGHTED[algo] and not weighted_copy:
        pytest.skip("needs weights")
    V, made, values = rows
    edges, dels = made[weighted_copy]
    directed = algo != "wcc"
    g = rg.Graph(V, len(edges), symmetric=not directed, weighted=weighted_copy)
    g.add_edges(edges, directed)
    g.del_edges(dels, directed)
    for k, v in {"dense_pull": 1, "bfs_bottom_up": 0, "pull_div": 1 << 30, "pull_split": split,
                 "pull_groups": groups, "cluster_edges": 0}.items():
        g.set_option(k, v)
    first, second = values(algo, weighted_copy)
    g.build_tree(algo, 0)
    np.testing.assert_array_equal(g.values(), first)
    g.add_edges(dels, directed)   # the copy, and the bounds of the groups, are rebuilt
    g.build_tree(algo, 0)
    np.testing.assert_array_equal(g.values(), second)
    g.close()


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("limit", [16384, 1 << 20])
def test_cluster_levels_in_profile_mode(algo, limit):
    """With one-CTA levels off, a launch that runs several levels is the cluster's.  A build, and batches on top of it."""
    scale = 14
    V = 1 << scale
    pairs = gen.rmat(scale, seed=71)
    imported = int(len(pairs) * 0.9)
    directed = algo != "wcc"
    root = 0 if algo == "wcc" else gen.max_out_degree_vertex(pairs[:imported], V)
    g = gpu_graph(algo, V, pairs[:imported], hint=len(pairs), inc_mode=True)
    og = oracle_graph(algo, V, pairs[:imported], inc_mode=True)
    for k, v in {"cluster_edges": limit, "tiny_edges": 0, "dense_pull": 0, "bfs_bottom_up": 0}.items():
        g.set_option(k, v)
    g.profile(True)
    g.build_tree(algo, root)
    og.build_tree(root)
    np.testing.assert_array_equal(g.values(), og.labels()[0])
    if limit == 1 << 20:   # every level fits (of WCC's four, 16,384 slots hold one)
        assert len(g.level_times()) < g.last_stats()["levels"]
    batch, nb = 2000, 4
    ref = og.run_batch(pairs, imported, batch, nb, root)
    e = edges_of(algo, pairs)
    for k in range(nb):
        lo = imported + k * batch
        g.apply_add(algo, e[lo:lo + batch], directed)
        g.apply_del(algo, e[lo - imported:lo - imported + batch], directed)
        assert g.checksum() == int(ref[k]), f"batch {k}"
    val, par, pw = g.labels()
    assert og.validate(val, par, pw, root) == 0
    g.close()


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("stepped", [False, True])
def test_heavy_vertices_in_the_loops_repair(algo, stepped):
    """The parent edges of the eight heaviest vertices go (lists longer than one warp takes): the rescue, expansion and
    pull of the queued vertices, from the cached graphs and stepped from the host."""
    scale = 16
    pairs = gen.rmat(scale, seed=91)
    V = 1 << scale
    directed = algo != "wcc"
    g = gpu_graph(algo, V, pairs, inc_mode=True)
    og = oracle_graph(algo, V, pairs, inc_mode=True)
    g.set_option("cluster_edges", 0)
    g.profile(stepped)
    root = gen.max_out_degree_vertex(pairs, V)
    g.build_tree(algo, root)
    og.build_tree(root)
    val, par, pw = g.labels()
    _, indeg = g.degrees()
    order = np.argsort(-indeg.astype(np.int64))
    hubs = [int(v) for v in order[:64] if par[v] != V and v != root][:8]
    assert len(hubs) == 8 and indeg[hubs[0]] > 2048
    one = np.zeros(len(hubs), rg.EDGE_DTYPE)
    one["src"], one["dst"] = par[hubs], hubs
    if WEIGHTED[algo]:
        one["data"] = pw[hubs]
    dels = np.repeat(one, np.maximum(g.get_edge_num(one), 1).astype(np.int64))
    g.apply_del(algo, dels, directed)
    old = np.array([og.del_edge(int(e["src"]), int(e["dst"]), int(e["data"])) for e in dels], np.uint64)
    gone = dels[old == 1]
    og.update_tree_del_batch(gone["src"], gone["dst"], gone["data"], root)
    val, par, pw = g.labels()
    np.testing.assert_array_equal(val, og.labels()[0])
    assert og.validate(val, par, pw, root) == 0
    g.close()
