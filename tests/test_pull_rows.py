"""Pull levels over rows of every kind the sliced in-edge copy holds: each list
length at which the copy's row kernels and the pull's slice classes change,
lists cut into pieces, tied and very large weights, and lists with deleted
entries, some of them whole lists.  Values equal the oracle's and trees are
valid, with the level in one launch, split, and in groups."""
import numpy as np
import pytest

import risgraph_b200 as rg
from oracle import oracle as O

from helpers import ALGOS, WEIGHTED

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 4, 5, 7, 8, 9, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 287, 288, 289, 575,
           576, 577, 1152, 1153, 1500]


def row_graph(seed):
    """(vertices, edges, edges deleted again): a sparse random graph over 2,000 vertices, and one vertex
    per length with that many in-edges from distinct ones of them, and an edge back."""
    rng = np.random.default_rng(seed)
    n = 2000
    V = n + 3 * len(LENGTHS)
    parts = [np.stack([rng.integers(0, n, 3 * n), rng.integers(0, n, 3 * n)], 1)]
    dels = []
    for k, length in enumerate(LENGTHS * 3):
        v = n + k
        e = np.stack([rng.permutation(n)[:length], np.full(length, v)], 1)
        parts += [e, np.array([[v, rng.integers(0, n)]])]
        if k >= 2 * len(LENGTHS):      # a third of these lists is deleted
            dels.append(e[rng.random(length) < 0.34])
        elif k % 7 == 0:               # and these whole
            dels.append(e)
    pairs = np.concatenate(parts).astype(np.uint64)
    edges = np.zeros(len(pairs), rg.EDGE_DTYPE)
    edges["src"], edges["dst"] = pairs[:, 0], pairs[:, 1]
    # weights: a function of the endpoints, so that a deleted edge names its weight
    w = (pairs[:, 0] * np.uint64(2654435761) + pairs[:, 1] * np.uint64(40503)) >> np.uint64(7)
    edges["data"] = np.choose((w % np.uint64(5)).astype(int),
                              [w % np.uint64(255) + np.uint64(1), w % np.uint64(3), np.full(len(w), 127, np.uint64),
                               np.uint64(128) + w % np.uint64(1 << 20), np.uint64((1 << 27) - 1) + w % np.uint64(3)])
    gone = {(int(s), int(d)) for part in dels for s, d in part}
    mask = np.fromiter(((int(s), int(d)) in gone for s, d in pairs), bool, len(pairs))
    return V, edges, edges[mask]


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("weighted_copy", [False, True])
@pytest.mark.parametrize("split,groups", [(0, 2), (1, 2), (1, 4)])
def test_pull_rows_of_every_length(algo, weighted_copy, split, groups):
    if WEIGHTED[algo] and not weighted_copy:
        pytest.skip("needs weights")
    V, edges, dels = row_graph(5)
    if not weighted_copy:
        edges, dels = edges.copy(), dels.copy()
        edges["data"] = 0
        dels["data"] = 0
    directed = algo != "wcc"
    g = rg.Graph(V, len(edges), symmetric=not directed, weighted=weighted_copy)
    g.add_edges(edges, directed)
    g.del_edges(dels, directed)
    for k, v in {"dense_pull": 1, "bfs_bottom_up": 0, "pull_div": 1 << 30, "pull_split": split,
                 "pull_groups": groups}.items():
        g.set_option(k, v)
    og = O.OracleGraph(algo, V, len(edges))
    for e in edges:
        og.add_edge(int(e["src"]), int(e["dst"]), int(e["data"]) if WEIGHTED[algo] else 0)
    for e in dels:
        og.del_edge(int(e["src"]), int(e["dst"]), int(e["data"]) if WEIGHTED[algo] else 0)
    root = 0
    og.build_tree(root)
    g.build_tree(algo, root)
    val, par, pw = g.labels()
    np.testing.assert_array_equal(val, og.labels()[0])
    if WEIGHTED[algo] or not weighted_copy:
        assert og.validate(val, par, pw, root) == 0
    # the copy is rebuilt after a change, in place
    g.add_edges(dels, directed)
    for e in dels:
        og.add_edge(int(e["src"]), int(e["dst"]), int(e["data"]) if WEIGHTED[algo] else 0)
    og.build_tree(root)
    g.build_tree(algo, root)
    np.testing.assert_array_equal(g.values(), og.labels()[0])
    g.close()
