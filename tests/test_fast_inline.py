"""Inline batches (up to 16 edges in the launch parameters) on graphs small
enough that every complication comes up: repeated edges in a batch, an edge both
inserted and deleted by one submission, self-loops, undirected pairs, lists that
have to grow, occupied index slots, deletes of what is not there, tree edges
deleted and replaced.  Multiplicities are counted on the host; the values and
trees are the oracle's after every few submissions."""
import collections

import numpy as np
import pytest

import risgraph_b200 as rg
from oracle import oracle as O

from helpers import ALGOS, WEIGHTED

pytestmark = pytest.mark.gpu


def edge_array(rows):
    e = np.zeros(len(rows), rg.EDGE_DTYPE)
    for k, f in enumerate(("src", "dst", "data")):
        e[f] = [r[k] for r in rows]
    return e


@pytest.mark.parametrize("algo", ALGOS)
@pytest.mark.parametrize("vertices,batch", [(6, 1), (6, 16), (40, 4), (40, 16), (700, 1), (700, 16)])
@pytest.mark.parametrize("dual", [False, True])
def test_inline_batches_vs_oracle(algo, vertices, batch, dual):
    if dual and algo != "wcc":
        pytest.skip("undirected updates of a graph with in-lists of its own: WCC only")
    directed, weighted = algo != "wcc", WEIGHTED[algo]
    rng = np.random.default_rng(vertices * 100 + batch)
    g = rg.Graph(vertices, 64, symmetric=not directed and not dual, weighted=weighted)
    count = collections.Counter()

    def draw(n, live):
        out = []
        keys = list(count)
        for _ in range(n):
            if live and keys and rng.random() < 0.7:
                out.append(keys[rng.integers(len(keys))])
            else:
                s, d = (int(x) for x in rng.integers(0, vertices, 2))
                w = int(rng.integers(1, 5)) if weighted else 0
                if not directed and s > d:
                    s, d = d, s
                out.append((s, d, w))
        return out

    def check():
        og = O.OracleGraph(algo, vertices, 64)
        for (s, d, w), n in count.items():
            for _ in range(n):
                og.add_edge(s, d, w)
        og.build_tree(0)
        val, par, pw = g.labels()
        np.testing.assert_array_equal(val, og.labels()[0])
        assert og.validate(val, par, pw, 0) == 0
        keys = [k for k in count if directed or k[0] != k[1]]
        if keys:
            np.testing.assert_array_equal(g.get_edge_num(edge_array(keys)), [count[k] for k in keys])

    g.build_tree(algo, 0)
    for step in range(60):
        adds, dels = draw(int(rng.integers(1, batch + 1)), False), draw(int(rng.integers(1, batch + 1)), True)
        if step % 3 == 0:
            old = g.apply_add(algo, edge_array(adds), directed)
            if len(adds) == 1 and (directed or adds[0][0] != adds[0][1]):
                assert int(old[0]) == count[adds[0]]
            for k in adds:
                count[k] += 1
            old = g.apply_del(algo, edge_array(dels), directed)
            if len(dels) == 1 and (directed or dels[0][0] != dels[0][1]):
                assert int(old[0]) == count[dels[0]]
        else:
            g.apply_add_del(algo, edge_array(adds), edge_array(dels), directed)
            for k in adds:
                count[k] += 1
        for k in dels:
            count[k] = max(0, count[k] - 1)
        if step % 4 == 3 or step > 55:
            check()
    g.close()
