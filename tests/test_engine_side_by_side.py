"""Repairs of several graphs at once, each from a thread of its own: batches on both
sides of the size up to which a repair takes half the SMs, with builds between
them.  Every graph keeps the values that it has alone."""
import threading

import numpy as np
import pytest

from risgraph_b200 import gen

from helpers import edges_of, gpu_graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(2049, 2049, 2049), (16384, 16385, 16384), (16385, 40_000, 3000)])
def test_repairs_side_by_side(sizes):
    scale = 15
    V = 1 << scale
    pairs = gen.rmat(scale, n_edges=16 * V, seed=31)
    root, n = gen.max_out_degree_vertex(pairs, V), 12 * V
    algos = ("sssp", "bfs", "sswp")
    graphs, want = [], []
    for algo, b in zip(algos, sizes):
        e = edges_of(algo, pairs)
        steps = [(e[n + k * b:n + (k + 1) * b], e[k * b:(k + 1) * b]) for k in range(2)]
        h = gpu_graph(algo, V, pairs[:n], hint=len(pairs))
        h.set_option("cluster_edges", 0)
        h.build_tree(algo, root)
        vals = []
        for adds, dels in steps + [(d, a) for a, d in reversed(steps)]:
            h.apply_add_del(algo, adds, dels)
            vals.append(h.values())
        h.close()
        graphs.append((gpu_graph(algo, V, pairs[:n], hint=len(pairs)), algo, steps))
        want.append(vals)
    bad = []

    def work(i):
        g, algo, steps = graphs[i]
        for r in range(6):
            if r % 3 == 0:
                g.build_tree(algo, root)
            for k, (adds, dels) in enumerate(steps + [(d, a) for a, d in reversed(steps)]):
                g.apply_add_del(algo, adds, dels)
                if not np.array_equal(g.values(), want[i][k]):
                    bad.append((algo, r, k))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(graphs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for g, _, _ in graphs:
        g.close()
