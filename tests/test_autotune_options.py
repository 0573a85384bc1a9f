"""The tuner settles an option where it has an effect: those that only the
graph-driven loop reads are its to choose when it chooses that loop, and stay as
they were when the grid engine stays on."""
import pytest

from risgraph_b200 import gen

from helpers import edges_of, gpu_graph

pytestmark = pytest.mark.gpu

# (neither is among the tuner's candidates)
OWN = {"dense_div": 33, "lbs_min": 3333}


@pytest.mark.parametrize("algo", ["bfs", "sssp"])
def test_options_of_the_loop_follow_the_loop(algo):
    """Single timings of a small graph, so that any setting wins now and then."""
    scale = 10
    V = 1 << scale
    pairs = gen.rmat(scale, seed=4)
    g = gpu_graph(algo, V, pairs)
    root = gen.max_out_degree_vertex(pairs, V)
    sample = edges_of(algo, pairs[:8])
    engine = g.get_option("cluster_edges")
    for _ in range(25):
        for k, v in {**OWN, "cluster_edges": engine}.items():
            g.set_option(k, v)
        got = g.autotune(algo, root, sample=sample, reps=1)["options"]
        assert got["cluster_edges"] in (0, engine)
        if got["cluster_edges"]:
            assert {k: got[k] for k in OWN} == OWN
    # a graph that is set to the loop may be given the engine, and keeps its own values then
    for _ in range(10):
        for k, v in {**OWN, "cluster_edges": 0}.items():
            g.set_option(k, v)
        got = g.autotune(algo, root, sample=sample, reps=1)["options"]
        assert got["cluster_edges"] in (0, engine)
        if got["cluster_edges"]:
            assert {k: got[k] for k in OWN} == OWN
    g.close()
