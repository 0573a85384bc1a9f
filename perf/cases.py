"""Performance cases of the framework: what a user's program does with it, timed end to end through the public API.

Each case is one of four things that the command-line drivers, the server and the benchmark do with a resident graph:

  build   a dependency tree from scratch over a loaded graph, and its values read back (the plain drivers)
  inc     sliding-window update batches, each inserting the next edges and deleting the oldest ones, and the values
          after them (the _inc drivers with batch 1, the _inc_batch drivers above)
  reload  a bulk insert and a bulk delete of a sixteenth of the graph, and then a build over what is left of it
  serve   a burst of single-edge updates through the server, its completions, and the values after it (_inc_rt)

Inputs are RMAT graphs (a/b/c = .57/.19/.19, duplicates and self-loops kept, seeded order), or half uniform and half
RMAT (`mix`); weights are splitmix64(src << 32 | dst) % 255 + 1, the root is the vertex of highest out-degree.  WCC takes
edges as undirected.  A graph of the update cases holds the first nine tenths of its edges.  Values are read into pinned
host memory.
"""
import math

import numpy as np
import torch

import risgraph_b200 as rg

WEIGHTED = {"bfs": False, "sssp": True, "sswp": True, "wcc": False}
ABC = (0.57, 0.19, 0.19)


def listed():
    """The cases, by what they stand for in use."""
    return [
        # the plain incremental driver: one update pair at a time on the benchmark's RMAT-16 graph
        dict(name="inc_bfs_v64k_b1", kind="inc", algo="bfs", vertices=1 << 16, edges=1 << 20, batch=1, steps=32, mix=False),
        # single updates of weighted shortest paths on a graph larger than L2
        dict(name="inc_sssp_v1m_b1", kind="inc", algo="sssp", vertices=1 << 20, edges=1 << 24, batch=1, steps=32, mix=False),
        # small batches, odd sizes
        dict(name="inc_sssp_v700k_b100", kind="inc", algo="sssp", vertices=700_001, edges=9_999_991, batch=100, steps=16,
             mix=False),
        # the heavy-deletion configuration's batch size: components that split and merge, undirected, mixed degrees
        dict(name="inc_wcc_v1m_b1000", kind="inc", algo="wcc", vertices=1 << 20, edges=1 << 22, batch=1000, steps=8, mix=True),
        # large batches of the batch driver
        dict(name="inc_sssp_v2m_b10k", kind="inc", algo="sssp", vertices=1 << 21, edges=1 << 25, batch=10_000, steps=4,
             mix=False),
        dict(name="inc_sswp_v1m_b100k", kind="inc", algo="sswp", vertices=1 << 20, edges=1 << 24, batch=100_000, steps=2,
             mix=False),
        # trees from scratch: the headline graph, the other algorithms, a small graph of ragged size
        dict(name="build_sssp_v4m", kind="build", algo="sssp", vertices=1 << 22, edges=1 << 26, batch=0, steps=1, mix=False),
        dict(name="build_bfs_v2m", kind="build", algo="bfs", vertices=1 << 21, edges=1 << 25, batch=0, steps=1, mix=False),
        dict(name="build_wcc_v1m", kind="build", algo="wcc", vertices=1 << 20, edges=1 << 24, batch=0, steps=1, mix=False),
        dict(name="build_sswp_v150k", kind="build", algo="sswp", vertices=150_001, edges=2_345_678, batch=0, steps=1, mix=False),
        # a graph that changes in bulk between two builds
        dict(name="reload_sssp_v1m", kind="reload", algo="sssp", vertices=1 << 20, edges=1 << 24, batch=1 << 20, steps=1,
             mix=False),
        # the served path: a burst of 8,192 update pairs to one instance
        dict(name="serve_sssp_v1m", kind="serve", algo="sssp", vertices=1 << 20, edges=1 << 24, batch=8192, steps=1, mix=False),
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the ranges above: any algorithm, sizes over their whole range, odd ones among them."""
    kind = rng.choice(["inc", "inc", "inc", "build", "build", "reload", "serve"])
    mix = rng.random() < 0.25
    vertices = _spread(rng, 20_000, 1 << 21)
    # (a mix with more edges is one component: sparser ones leave components to maintain)
    edges = vertices * (rng.randint(2, 6) if mix else rng.randint(8, 16)) + rng.randint(0, 999)
    batch, steps = 0, 1
    if kind == "inc":
        batch = _spread(rng, 1, max(1, min(100_000, edges // 100)))
        steps = max(1, min(32, int(32 / max(1.0, math.sqrt(batch / 4.0)))))
    elif kind == "reload":
        batch = edges // 16
    elif kind == "serve":
        batch = _spread(rng, 500, min(16_384, edges // 32))
    return dict(kind=kind, algo=rng.choice(list(WEIGHTED)), vertices=vertices, edges=edges, batch=batch, steps=steps,
                mix=mix)


def _splitmix64(x):
    """splitmix64 of int64 tensors, taken as unsigned words."""
    def shr(v, k):
        return (v >> k) & ((1 << (64 - k)) - 1)

    z = x - 0x61C8864680B583EB  # + 0x9E3779B97F4A7C15
    z = (z ^ shr(z, 30)) * -0x40A7B892E31B1A47  # * 0xBF58476D1CE4E5B9
    z = (z ^ shr(z, 27)) * -0x6B2FB644ECCEEE15  # * 0x94D049BB133111EB
    return z ^ shr(z, 31)


def _weights(pairs):
    """splitmix64(src << 32 | dst) % 255 + 1 (2^64 % 255 is 1, so a negative word counts one more)."""
    z = _splitmix64((pairs[:, 0] << 32) | pairs[:, 1])
    return (torch.remainder(z, 255) + (z < 0)) % 255 + 1


def _pairs(case, seed):
    """The case's (edges, 2) int64 edge list, on the GPU."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n, v = case["edges"], case["vertices"]
    a, b, c = ABC
    src = torch.zeros(n, dtype=torch.int64, device="cuda")
    dst = torch.zeros(n, dtype=torch.int64, device="cuda")
    for _ in range(max(1, (v - 1).bit_length())):
        r = torch.rand(n, device="cuda", generator=gen)
        src = src * 2 + (r >= a + b)
        dst = dst * 2 + (((r >= a) & (r < a + b)) | (r >= a + b + c))
    pairs = torch.stack((src % v, dst % v), 1)
    if case["mix"]:
        half = torch.randint(0, v, ((n + 1) // 2, 2), device="cuda", generator=gen)
        pairs[::2] = half
    return pairs


def _root(pairs, v):
    deg = torch.bincount(pairs[:, 0], minlength=v)
    return int((deg == deg.max()).nonzero()[0])


def _loaded(case):
    """Edges that the graph holds before a pass."""
    e = case["edges"]
    return e if case["kind"] == "build" else e - e // 16 if case["kind"] == "reload" else e - e // 10


def _host_pairs(pairs):
    return pairs.cpu().numpy().view(np.uint64)


def _host_edges(pairs, weighted):
    """The pairs as an array of the library's edge records."""
    w = _weights(pairs) if weighted else torch.zeros_like(pairs[:, 0])
    return torch.cat((pairs, w[:, None]), 1).cpu().numpy().view(rg.EDGE_DTYPE).reshape(-1)


def prepare(case, seed):
    algo, v, kind = case["algo"], case["vertices"], case["kind"]
    pairs = _pairs(case, seed)
    root = _root(pairs, v)
    n, directed = _loaded(case), algo != "wcc"
    g = rg.Graph(v, len(pairs), symmetric=not directed, weighted=WEIGHTED[algo])
    g.add_pairs(_host_pairs(pairs[:n]), directed, want_old=False)
    state = {"case": case, "graph": g, "root": root, "directed": directed, "at": 0,
             "values": torch.empty(v, dtype=torch.int64, pin_memory=True)}
    if kind in ("inc", "serve"):
        # the edges that slide in and those that slide out, a whole number of batches of each
        k = (len(pairs) - n) // case["batch"] * case["batch"]
        state["in"], state["out"] = (_host_edges(p, WEIGHTED[algo]) for p in (pairs[n:n + k], pairs[:k]))
        g.build_tree(algo, root)
    elif kind == "reload":
        k = len(pairs) - n
        state["in"], state["out"] = _host_pairs(pairs[n:]), _host_pairs(pairs[:k])
    if kind == "serve":
        state["server"] = rg.Server()
    return state


def _next(state):
    """The next edges to insert and to delete; at the end of the stream the two lists change places."""
    b = state["case"]["batch"]
    if state["at"] + b > len(state["in"]):
        state["in"], state["out"], state["at"] = state["out"], state["in"], 0
    k = state["at"]
    state["at"] = k + b
    return state["in"][k:k + b], state["out"][k:k + b]


def _values(state):
    out = state["values"]
    status = rg.lib().rg_get_labels(state["graph"]._h, out.data_ptr(), None, None)
    if status:
        raise rg.RGError(status, "rg_get_labels")
    return out


def _requests(instance, adds, dels):
    """An insert and a delete by turns, as a sliding window's client sends them."""
    r = np.zeros(2 * len(adds), rg.REQUEST_DTYPE)
    r["instance"] = instance
    for k, e in ((0, adds), (1, dels)):
        r["type"][k::2] = k
        for f in ("src", "dst", "data"):
            r[f][k::2] = e[f]
    r["tag"] = np.arange(len(r))
    return r


def run(state):
    case, g, algo = state["case"], state["graph"], state["case"]["algo"]
    if case["kind"] == "build":
        g.build_tree(algo, state["root"])
        return _values(state)
    if case["kind"] == "reload":
        adds, dels = _next(state)
        g.add_pairs(adds, state["directed"], want_old=False)
        g.del_pairs(dels, state["directed"], want_old=False)
        g.build_tree(algo, state["root"])
        return _values(state)
    if case["kind"] == "serve":
        server = state["server"]
        instance = server.attach(g, state["directed"])
        server.submit(_requests(instance, *_next(state)))
        server.drain()
        done = server.poll()
        server.detach(instance)
        order = np.argsort(done["tag"])
        return {"values": _values(state), "tag": done["tag"][order].astype(np.int64), "status": done["status"][order],
                "type": done["type"][order].astype(np.int64)}
    for _ in range(case["steps"]):
        adds, dels = _next(state)
        g.apply_add_del(algo, adds, dels, state["directed"])
    return _values(state)


def work(case):
    """Bytes of one pass: each edge that a build reads once (4 bytes, 8 with a weight), each update record that comes in
    once, each value that goes out once."""
    directed, weighted = case["algo"] != "wcc", WEIGHTED[case["algo"]]
    edge = (8 if weighted else 4) * (1 if directed else 2)
    out = 8 * case["vertices"]
    if case["kind"] == "build":
        return {"bytes": case["edges"] * edge + out, "flops": 0}
    if case["kind"] == "reload":
        return {"bytes": _loaded(case) * edge + 2 * 16 * case["batch"] + out, "flops": 0}
    record = 40 + 48 if case["kind"] == "serve" else 24
    return {"bytes": 2 * record * case["batch"] * case["steps"] + out, "flops": 0}


def exact(case, seed):
    """The values by plain relaxation over the edges that the graph holds after the pass."""
    algo, v = case["algo"], case["vertices"]
    pairs = _pairs(case, seed)
    root = _root(pairs, v)
    n = _loaded(case)
    k = case["batch"] * case["steps"]
    live = pairs[k:n + k]
    src, dst = live[:, 0].contiguous(), live[:, 1].contiguous()
    if algo == "wcc":
        src, dst = torch.cat((src, dst)), torch.cat((dst, src))
        val = torch.arange(v, device="cuda")
    else:
        val = torch.full((v,), {"bfs": 65536, "sssp": 1 << 27, "sswp": 0}[algo], dtype=torch.int64, device="cuda")
        val[root] = 1 << 27 if algo == "sswp" else 0
    w = _weights(live) if WEIGHTED[algo] else None
    while True:
        new = val[src]
        if algo == "bfs":
            new = new + 1
        elif algo == "sssp":
            new = new + w
        elif algo == "sswp":
            new = torch.minimum(new, w)
        best = val.scatter_reduce(0, dst, new, "amax" if algo == "sswp" else "amin")
        if torch.equal(best, val):
            break
        val = best
    if case["kind"] == "serve":
        m = 2 * case["batch"]
        tag = torch.arange(m)
        return {"values": val, "tag": tag, "status": torch.zeros(m, dtype=torch.int32), "type": tag % 2}
    return val
