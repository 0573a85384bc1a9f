"""Staging of large batches: sizes on both sides of the staging step and of the
parallel pass, a fault anywhere in a batch (or in the second batch of a
submission) leaves the graph as it was, and weights that need codes are found
wherever they are."""
import numpy as np
import pytest

import risgraph_b200 as rg
from risgraph_b200 import gen

pytestmark = pytest.mark.gpu

STEP = 1 << 18


@pytest.mark.parametrize("n", [2049, STEP - 1, STEP, STEP + 1, 2 * STEP + 17])
@pytest.mark.parametrize("weighted", [False, True])
def test_large_batches_and_faults(n, weighted):
    V = 50_000
    pairs = gen.rmat(16, n, seed=n) % V
    e = gen.edges_with_weights(pairs, weighted)
    g = rg.Graph(V, 2 * n, weighted=weighted)
    g.add_pairs(pairs)
    out_deg, in_deg = g.degrees()
    np.testing.assert_array_equal(out_deg, np.bincount(pairs[:, 0].astype(int), minlength=V))
    np.testing.assert_array_equal(in_deg, np.bincount(pairs[:, 1].astype(int), minlength=V))
    g.build_tree("bfs", 0)
    before = g.checksum()
    for at in (0, n // 2, n - 1):
        for bad_id in (V, (1 << 63) + 1, (1 << 64) - 1):
            bad = e.copy()
            bad["dst"][at] = bad_id
            for call in (lambda: g.add_edges(bad), lambda: g.apply_del("bfs", bad),
                         lambda: g.apply_add_del("bfs", e, bad), lambda: g.add_pairs(bad.view(np.uint64).reshape(-1, 3)[:, :2])):
                with pytest.raises(rg.RGError) as err:
                    call()
                assert err.value.status == 2
    if weighted:
        bad = e.copy()
        bad["data"][n - 1] = (1 << 64) - (1 << 27)
        with pytest.raises(rg.RGError) as err:
            g.apply_add_del("bfs", e, bad)
        assert err.value.status == 3
    np.testing.assert_array_equal(g.degrees()[0], out_deg)   # nothing was applied
    assert g.checksum() == before
    if weighted:
        big = e.copy()
        big["data"][n - 1] = 1 << 40
        old = g.add_edges(big)
        assert old[n - 1] == 0 and g.get_edge_num(big[n - 1:])[0] == 1
        assert (old[:n - 1] > 0).all()
        g.del_edges(big)
    # an insert and a delete batch of these sizes, back to where it was
    g.apply_add_del("bfs", e, e)
    np.testing.assert_array_equal(g.degrees()[0], out_deg)
    assert g.checksum() == before
    g.close()
