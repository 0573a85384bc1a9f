"""Directed and undirected updates mixed on one graph, so that the two orientations
of an undirected edge have different multiplicities.  The count that decides and
comes back is that of the orientation with the lower source, whichever way round
the caller names the edge (the lower one's old count, core/graph.hpp:206-211,
:232-237, as both orientations count alike when every update is undirected); a
batch in the launch parameters answers as the staged phases do."""
import itertools

import numpy as np
import pytest

import risgraph_b200 as rg

pytestmark = pytest.mark.gpu


def edge(s, d, w=3):
    e = np.zeros(1, rg.EDGE_DTYPE)
    e["src"], e["dst"], e["data"] = s, d, w
    return e


def answers(algo, symmetric, pre, und, inline_max):
    weighted = algo == "sssp"
    g = rg.Graph(8, 64, symmetric=symmetric, weighted=weighted)
    g.set_option("inline_max", inline_max)
    g.add_edges(np.concatenate([edge(0, 3), edge(0, 1), edge(1, 5)]), True)
    g.build_tree(algo, 0)
    out = []

    def note(*old):
        out.extend(int(x) for o in old for x in o)
        out.extend(int(x) for x in g.values())
        out.extend(int(x) for x in g.get_edge_num(np.concatenate([edge(2, 3), edge(3, 2)])))

    note(g.apply_add(algo, edge(*pre), True))
    for _ in range(2):
        note(g.apply_add(algo, edge(*und), False))
    note(g.apply_del(algo, edge(*und), False))
    note(g.apply_del(algo, edge(*pre), True))
    note(g.apply_add(algo, edge(*und), False))
    for _ in range(3):
        note(g.apply_del(algo, edge(*und), False))
    g.apply_add(algo, edge(*pre), True)
    g.apply_add_del(algo, edge(*und), edge(1, 5), False)
    note()
    g.apply_add_del(algo, edge(6, 5), edge(*und), False)
    note()
    g.close()
    return out


@pytest.mark.parametrize("algo,symmetric", [("bfs", False), ("sssp", False), ("wcc", False), ("wcc", True)])
@pytest.mark.parametrize("pre,und", list(itertools.product([(2, 3), (3, 2)], repeat=2)))
def test_inline_batches_answer_as_the_phases(algo, symmetric, pre, und):
    assert answers(algo, symmetric, pre, und, 16) == answers(algo, symmetric, pre, und, 0)
