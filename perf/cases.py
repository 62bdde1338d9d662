"""The work a user has this framework do, as timed cases over its public entry points.

Kinds of case (`"kind"`):

  bfs        one BFS from one root on a resident graph, every entry of pred written (run_bfs; the
             direction-optimizing search the Graph500 benchmark times 64 times per graph)
  msbfs      one call of the batched form: up to 128 roots, a uint8 level row per root
  serve      a burst of queries to the request loop over several resident graphs, each query's
             levels delivered to a buffer of its own
  generate   a range of the Kronecker edge list (spec 2010 or 2012) into device memory
  construct  a graph built from a device edge list, used for one BFS and given back: the start-up
             of a benchmark run
  iteration  one root of the benchmark's main loop: run_bfs, then the Graph500 validator on its result
             against the graph's edge list

Every output is whole numbers that any correct implementation returns alike, so every tolerance is
"exact" and there are no computed floating-point outputs to hold against 64-bit ones.  The one
result that is free is which of several parents of the same level pred names; a BFS case therefore
returns the level field of every pred entry (a view of pred, no pass over it) with the counts that
run_bfs reports, and the iteration cases what the validator says about the parents as well.
"""
import numpy as np
import torch

import graph500_b200 as g5

# the direction settings in use: the reference's thresholds (the default), the setting the autotuner
# settles on for Kronecker graphs (bottom-up to the end), and the edge-count policy
SETTINGS = {"default": (2000.0, 8.0, g5.DIR_REFERENCE), "tuned": (2000.0, 1e9, g5.DIR_REFERENCE),
            "edges": (15.0, 24.0, g5.DIR_EDGES)}


def listed():
    M = 1 << 20
    return [
        # the smallest of the benchmark's configurations: launch and barrier latency
        {"name": "bfs-s16-vr0", "kind": "bfs", "scale": 16, "edges": M, "vr": 0, "setting": "default", "pred": "device"},
        # the reference driver's own call: pred in plain host memory
        {"name": "bfs-s21-host", "kind": "bfs", "scale": 21, "edges": 32 * M, "vr": 2, "setting": "default",
         "pred": "host"},
        # the headline configuration, with the setting its autotuner picks
        {"name": "bfs-s22", "kind": "bfs", "scale": 22, "edges": 64 * M, "vr": 2, "setting": "tuned", "pred": "device"},
        # past L2, with the default thresholds (the search turns back to top-down at its end)
        {"name": "bfs-s24", "kind": "bfs", "scale": 24, "edges": 256 * M, "vr": 2, "setting": "default",
         "pred": "device"},
        # the largest configuration of the benchmark
        {"name": "bfs-s26", "kind": "bfs", "scale": 26, "edges": 1024 * M, "vr": 2, "setting": "tuned",
         "pred": "device"},
        # a small batch on a small graph, with each root's edge count: what a server launches most
        {"name": "msbfs-s18-r24", "kind": "msbfs", "scale": 18, "edges": 4 * M, "vr": 2, "roots": 24, "lanes": 32,
         "levels": "resident", "stats": True},
        # the widest batch, levels copied to the caller's device buffer
        {"name": "msbfs-s21-r128", "kind": "msbfs", "scale": 21, "edges": 32 * M, "vr": 2, "roots": 128, "lanes": 128,
         "levels": "device", "stats": False},
        # the batched configuration of the benchmark: 64 roots, levels left on the device
        {"name": "msbfs-s24-r64", "kind": "msbfs", "scale": 24, "edges": 256 * M, "vr": 2, "roots": 64, "lanes": 64,
         "levels": "resident", "stats": False},
        # a burst of queries over resident graphs of different sizes
        {"name": "serve-3-graphs", "kind": "serve", "scales": "18,20,22", "queries": 192},
        # an edge list on the device
        {"name": "generate-s22", "kind": "generate", "scale": 22, "edges": 64 * M, "spec": 2010},
        # a graph from its edge list, degree-sorted, to the first BFS
        {"name": "construct-s22", "kind": "construct", "scale": 22, "edges": 64 * M, "vr": 2},
        # one root of the benchmark's loop, search and validation, on a graph past L2
        {"name": "iteration-s24", "kind": "iteration", "scale": 24, "edges": 256 * M, "vr": 2, "setting": "default"},
    ]


def _edges(rng, scale, most=1 << 30):
    """An odd number of edges, between 6 and 24 per vertex id."""
    return min(most, int((1 << scale) * rng.uniform(6, 24))) | 1


def draw(rng):
    kind = rng.choice(["bfs", "bfs", "bfs", "msbfs", "msbfs", "serve", "generate", "construct", "iteration"])
    if kind == "bfs":
        scale = rng.randint(12, 25)
        vr = 2 if scale > 21 else rng.choice([0, 1, 2, 2])
        pred = rng.choice(["device", "device", "host", "pinned"]) if scale <= 22 else "device"
        return {"kind": kind, "scale": scale, "edges": _edges(rng, scale), "vr": vr,
                "setting": rng.choice(sorted(SETTINGS)), "pred": pred}
    if kind == "msbfs":
        scale = rng.randint(14, 23)
        return {"kind": kind, "scale": scale, "edges": _edges(rng, scale), "vr": 2 if scale > 20 else rng.choice([0, 1, 2, 2]),
                "roots": rng.randint(1, 128), "lanes": rng.choice([32, 64, 128]),
                "levels": rng.choice(["resident", "device", "host"] if scale < 21 else ["resident", "device"]),
                "stats": False}
    if kind == "serve":
        scales = sorted(rng.randint(13, 21) for _ in range(rng.randint(1, 3)))
        return {"kind": kind, "scales": ",".join(map(str, scales)), "queries": int(2 ** rng.uniform(3, 8)) | 1}
    if kind == "generate":
        scale = rng.randint(12, 26)
        return {"kind": kind, "scale": scale, "edges": int(2 ** rng.uniform(16, min(scale + 4, 27))) | 1,
                "spec": rng.choice([2010, 2010, 2012])}
    if kind == "construct":
        scale = rng.randint(12, 23)
        return {"kind": kind, "scale": scale, "edges": _edges(rng, scale), "vr": rng.choice([0, 1, 2, 2])}
    scale = rng.randint(12, 25)
    return {"kind": kind, "scale": scale, "edges": _edges(rng, scale), "vr": 2, "setting": rng.choice(sorted(SETTINGS))}


class State:
    """What a program holds before the call; handles are given back before the graphs they belong to."""

    def __init__(self, case):
        self.case = case
        self.handles = []

    def __del__(self):
        for h in reversed(self.handles):
            h.close()


def _edge_list(scale, edges, seed):
    """The first `edges` edges of a Kronecker graph in device memory."""
    out = torch.empty((edges, 3), dtype=torch.int32, device="cuda")
    g5.generate_edges(scale, -(-edges >> scale), 0, edges, seed + 2, 3, out)
    return out


def _graph(case, seed, keep_edges=False):
    bfs = g5.BfsOnGPU(reorder_mode=case["vr"])
    edges = _edge_list(case["scale"], case["edges"], seed)
    bfs.construct(edges, keep_edges=keep_edges)
    return bfs, edges


def _roots(graph, n, seed):
    return g5.find_roots(graph, n, seed + 5, 7)


def prepare(case, seed):
    s = State(case)
    kind = case["kind"]
    if kind == "generate":
        s.seed = seed
        s.start = (seed * 7919) % (1 << case["scale"]) if case["spec"] == 2010 else 0
        words = 3 if case["spec"] == 2010 else 4
        s.out = torch.empty((case["edges"], words), dtype=torch.int32, device="cuda")
        s.edgefactor = -(-(s.start + case["edges"]) >> case["scale"])
    elif kind == "construct":
        s.edges = _edge_list(case["scale"], case["edges"], seed)
        s.pred = torch.empty(max(1 << case["scale"], 1 << 16), dtype=torch.int64, device="cuda")
        s.seed = seed
    elif kind == "serve":
        graphs, s.queries = [], []
        for i, scale in enumerate(int(x) for x in case["scales"].split(",")):
            g = g5.Graph2DCSR.generate(scale, 16, 2, 0, seed + 2 + i, 3)
            s.handles.append(g)
            graphs.append(g)
        s.server = g5.Server(graphs)
        s.handles.append(s.server)
        rng = np.random.default_rng(seed)
        which = rng.permutation(np.arange(case["queries"]) % len(graphs))
        s.levels = [torch.empty((int(np.sum(which == i)), g.pred_size()), dtype=torch.uint8, device="cuda")
                    for i, g in enumerate(graphs)]
        taken = [0] * len(graphs)
        roots = [_roots(g, int(np.sum(which == i)), seed) for i, g in enumerate(graphs)]
        for i in which:
            k = taken[i]
            taken[i] += 1
            s.queries.append((int(i), int(roots[i][k]), s.levels[i][k]))
    else:
        s.bfs, edges = _graph(case, seed, keep_edges=kind == "iteration")
        s.handles.append(s.bfs)
        graph = s.bfs.graph_
        if kind == "msbfs":
            s.roots = _roots(graph, case["roots"], seed)
            s.ms = g5.MultiSourceBFS(graph, case["lanes"])
            s.handles.append(s.ms)
            s.levels = None
            if case["levels"] == "device":
                s.levels = torch.empty((case["roots"], graph.pred_size()), dtype=torch.uint8, device="cuda")
            elif case["levels"] == "host":
                s.levels = torch.empty((case["roots"], graph.pred_size()), dtype=torch.uint8, pin_memory=True).numpy()
        else:
            alpha, beta, policy = SETTINGS[case["setting"]]
            s.bfs.prepare_bfs(alpha, beta, False, policy)
            s.root = int(_roots(graph, 1, seed)[0])
            n = graph.pred_size()
            if case.get("pred", "device") == "device":
                s.pred = torch.empty(n, dtype=torch.int64, device="cuda")
            elif case["pred"] == "pinned":
                s.pred = torch.empty(n, dtype=torch.int64, pin_memory=True).numpy()
            else:
                s.pred = np.zeros(n, np.int64)
            s.edges = edges if kind == "iteration" else None  # the validator reads the caller's list
    return s


def _levels_of(pred):
    """The level field of every pred entry (-1 unreached), as a view."""
    if isinstance(pred, np.ndarray):
        return pred.view(np.int16)[3::4]
    return pred.view(torch.int16).view(-1, 4)[:, 3]


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "bfs":
        st = s.bfs.run_bfs(s.root, s.pred)
        return _levels_of(s.pred), st.reached, st.nedge, st.num_levels
    if kind == "msbfs":
        st = s.ms.run(s.roots, s.levels)
        levels = s.levels
        if levels is None:
            levels = s.ms.device_levels(len(s.roots))  # a view of the handle's own memory:
            levels.owner = s                           # the handle lives as long as it does
        out = [levels, st.num_levels]
        if case["stats"]:
            out += s.ms.root_stats(len(s.roots))
        return out
    if kind == "serve":
        for i, (g, root, levels) in enumerate(s.queries):
            s.server.submit(g, root, i, levels)
        s.server.drain()
        done = sorted(s.server.poll(len(s.queries)), key=lambda r: r["tag"])
        return s.levels, np.array([(r["tag"], r["status"], r["reached"], r["nedge"]) for r in done])
    if kind == "generate":
        f = g5.generate_edges if case["spec"] == 2010 else g5.generate_edges_spec2012
        f(case["scale"], s.edgefactor, s.start, s.start + case["edges"], s.seed + 2, 3, s.out)
        return s.out
    if kind == "construct":
        bfs = g5.BfsOnGPU(reorder_mode=case["vr"])
        bfs.construct(s.edges, keep_edges=False)
        info = bfs.graph_.info
        roots = g5.find_roots(bfs.graph_, 64)
        bfs.prepare_bfs()
        st = bfs.run_bfs(int(roots[0]), s.pred)
        scalars = [info.pred_size, info.num_local_verts, info.num_global_verts, info.num_global_edges,
                   info.max_used_vertex, st.reached, st.nedge, st.num_levels]
        bfs.close()
        return _levels_of(s.pred), roots, scalars
    st = s.bfs.run_bfs(s.root, s.pred)
    ok, visited, report = g5.validate_bfs_result(s.bfs.graph_, s.root, s.pred)
    return _levels_of(s.pred), st.reached, st.nedge, ok, visited, report


def work(case):
    """Inputs read once and outputs written once.  A BFS has to read one adjacency entry per vertex id (its
    parent's) and write its pred entry; the batched form reads the adjacency once for all its roots."""
    kind = case["kind"]
    if kind == "serve":
        sizes = [1 << int(x) for x in case["scales"].split(",")]
        return {"bytes": sum(8 * 16 * n + case["queries"] // len(sizes) * n for n in sizes), "flops": 0}
    n, m = 1 << case["scale"], case["edges"]
    if kind == "bfs":
        return {"bytes": 8 * n + 4 * n, "flops": 0}
    if kind == "msbfs":
        return {"bytes": case["roots"] * n + 8 * m, "flops": 0}
    if kind == "generate":
        return {"bytes": (12 if case["spec"] == 2010 else 16) * m, "flops": 0}
    if kind == "construct":  # edges in; two adjacency entries per edge, row starts, three maps and pred out
        return {"bytes": 12 * m + 8 * m + 8 * n + 12 * n + 8 * n, "flops": 0}
    return {"bytes": 12 * m + 8 * n + 4 * n, "flops": 0}


def tolerance(case):
    return "exact"
