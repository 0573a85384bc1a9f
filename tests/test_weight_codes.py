"""Weights above 2^27 travel as codes that the graph remembers: a submission that is
refused leaves none behind."""
import os

import numpy as np
import pytest

import risgraph_b200 as rg

pytestmark = pytest.mark.gpu


def resident_mb():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * os.sysconf("SC_PAGE_SIZE") / 2**20


def test_a_refused_submission_leaves_no_codes():
    V, n, calls = 1000, 400_000, 8
    g = rg.Graph(V, 2 * n, weighted=True)
    g.build_tree("sssp", 0)
    e = np.zeros(n, rg.EDGE_DTYPE)
    e["src"], e["dst"] = np.arange(n) % V, np.arange(n) // V % V
    bad = e[:3000].copy()
    bad["dst"][2999] = V

    def refused(k):
        e["data"] = (1 << 40) + k * n + np.arange(n)   # every weight a new one
        with pytest.raises(rg.RGError) as err:
            g.apply_add_del("sssp", e, bad)
        assert err.value.status == 2

    for k in range(2):
        refused(k)
    at = resident_mb()
    for k in range(2, 2 + calls):
        refused(k)
    # a code takes a table entry, a node and a list entry: 40 bytes at the least
    assert resident_mb() - at < calls * n * 40 / 2**20 / 2
    assert (g.degrees()[0] == 0).all()
    # and an accepted one reads back whole
    e["data"] = (1 << 40) + np.arange(n)
    g.apply_add_del("sssp", e, bad[:1])
    assert g.get_edge_num(e[-1:])[0] == 1
    g.close()
