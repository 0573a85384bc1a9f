"""Edge lookup of insert batches in a nearly full edge index: probe runs longer
than one step, runs that wrap around the end of the index, keys repeated within
a warp and across warps of one batch, keys that exist already, deletes of keys
that do not.  The index of a graph with a small edge hint has 2,048 slots and 1,792
records, and 1,600 keys fill it to 78%; multiplicities are counted on the host.
(Two ops of one batch that insert the same new key may use up a record each, so
a batch repeats few of its new keys.)"""
import collections

import numpy as np
import pytest

import risgraph_b200 as rg

pytestmark = pytest.mark.gpu

V = 40  # 1,600 keys


@pytest.mark.parametrize("algo", ["bfs", "sssp"])
@pytest.mark.parametrize("fused_max", [2048, 16])
@pytest.mark.parametrize("batch", [1, 17, 31, 33, 255, 1000, 1600])
def test_lookup_in_a_dense_index(algo, fused_max, batch):
    rng = np.random.default_rng(batch)
    g = rg.Graph(V, 64, weighted=algo == "sssp")
    g.set_option("fused_max", fused_max)
    keys = np.zeros(0, np.int64)
    g.build_tree(algo, 0)
    count = collections.Counter()
    for _ in range(12):
        while len(keys) < batch:
            keys = np.concatenate([keys, rng.permutation(V * V)])
        take, keys = keys[:batch].copy(), keys[batch:]
        take[: batch // 16] = rng.integers(0, 4, batch // 16)  # neighbours in the batch share a key
        take[batch // 2 :: 37] = take[0]  # and lanes of several warps
        adds = np.zeros(batch, rg.EDGE_DTYPE)
        adds["src"], adds["dst"] = np.divmod(take, V)
        dels = adds[rng.random(batch) < 0.3].copy()
        if len(dels):
            dels["src"][0], dels["dst"][0] = V - 1, rng.integers(0, V)
        g.apply_add_del(algo, adds, dels, True)
        for e in adds:
            count[(int(e["src"]), int(e["dst"]))] += 1
        for e in dels:
            k = (int(e["src"]), int(e["dst"]))
            count[k] = max(0, count[k] - 1)
        q = np.zeros(V * V, rg.EDGE_DTYPE)
        q["src"], q["dst"] = np.divmod(np.arange(V * V), V)
        want = np.array([count[(int(s), int(d))] for s, d in zip(q["src"], q["dst"])])
        np.testing.assert_array_equal(g.get_edge_num(q), want)
    g.close()
