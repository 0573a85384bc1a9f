"""BFS builds that may both pull (RG_OPT_DENSE_PULL 1) and go bottom-up: a pull level
commits values deeper than the level, so a bottom-up level, which looks for
parents of one depth, must not follow it."""
import numpy as np
import pytest

import risgraph_b200 as rg

pytestmark = pytest.mark.gpu

KIDS, MID = 2100, 300_000


def layered_pairs():
    """The root, its KIDS children, MID vertices with eight parents among them, one child of each of these (a shorter
    list, pulled after it), and one child of every third of those."""
    kids = 1 + np.arange(KIDS)
    mid = kids[-1] + 1 + np.arange(MID)
    low = mid + MID
    leaf = low[-1] + 1 + np.arange(MID // 3)
    deep = np.stack([kids[(np.arange(8 * MID) * 37 + np.arange(8 * MID) // MID) % KIDS], np.tile(mid, 8)], 1)
    pairs = np.concatenate([np.stack([np.zeros(KIDS, int), kids], 1), deep, np.stack([mid, low], 1),
                            np.stack([low[:len(leaf)], leaf], 1)])
    depth = np.concatenate([[0], np.full(KIDS, 1), np.full(MID, 2), np.full(MID, 3), np.full(len(leaf), 4)])
    return pairs.astype(np.uint64), depth.astype(np.uint64)


@pytest.mark.parametrize("cluster_edges", [0, 65536])
@pytest.mark.parametrize("pull_div", [64, 1 << 30])
def test_values_are_the_depths(cluster_edges, pull_div):
    pairs, depth = layered_pairs()
    g = rg.Graph(len(depth), len(pairs))
    g.add_pairs(pairs, want_old=False)
    for k, v in {"dense_pull": 1, "pull_div": pull_div, "cluster_edges": cluster_edges}.items():
        g.set_option(k, v)
    for _ in range(3):
        g.build_tree("bfs", 0)
        np.testing.assert_array_equal(g.values(), depth)
    g.close()
