"""Performance cases: what programs have this framework do, through its public
entry points, from the smallest graphs to the largest that three copies of
fit one GPU.

Graphs are Kronecker graphs with the Graph500 initiator (0.57, 0.19, 0.19,
0.05) and uniform [0, 1) weights, generated here with plain torch, so that the
inputs, and the exact distances, do not depend on the framework's own
generator; vertex counts need not be powers of two.  Roots are uniform over
the vertices within two hops of the highest-degree vertex, i.e. in the giant
component, as nearly all of the benchmark's roots are.

Kinds of case:
  generate    the benchmark's edge generator over a range of edges
  build       the graph of an edge list: the canonical CSR and the copies that
              the searches read
  bfs_query   one synchronous search of a resident graph, statistics on the host
  bfs         one search, enqueued (reset and traversal)
  sssp        one shortest-path search, enqueued
  runner      the benchmark's protocol for one root: both searches, distances
              from the parents, both validations and the edge count
  msbfs       a batch of up to 256 searches of one graph, depths as bytes
  sssp_multi  a batch of up to 32 shortest-path searches of one graph
  packed      one BFS and one SSSP of each of many small graphs at once

BFS parents are not among the outputs: every tree edge of a shortest path is a
right one, and which is found depends on the order of atomics.  The depths
are unique; `runner` returns the distances that the framework derives from
the parents, and the validation's error counts.
"""
import importlib.util
import os
import sys

import numpy as np
import torch

_REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_NAME = "cgt_b200"  # the package's folder name is not an identifier


def _package():
    if _NAME not in sys.modules:
        folder = os.path.join(_REPO, "cuda-graph-traversal_b200")
        spec = importlib.util.spec_from_file_location(_NAME, os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[_NAME] = mod
        spec.loader.exec_module(mod)
    return sys.modules[_NAME]


G = _package()
DEV = "cuda"


# ------------------------------------------------------------------ cases ----

def listed():
    return [
        # One interactive query of a SCALE 12 graph: launches and the host's
        # wait are all of it.
        {"name": "bfs query, 4 K vertices", "kind": "bfs_query", "n": 1 << 12, "ef": 16},
        # A search of an ordinary graph whose vertex count is not a power of two.
        {"name": "bfs, 700 K vertices", "kind": "bfs", "n": 700_001, "ef": 16},
        # The largest search: 1.07 G CSR entries.
        {"name": "bfs, 34 M vertices", "kind": "bfs", "n": 1 << 25, "ef": 16},
        # Shortest paths on a small graph, where phases and barriers count.
        {"name": "sssp, 16 K vertices", "kind": "sssp", "n": 1 << 14, "ef": 16},
        # An ordinary one, with an odd vertex count.
        {"name": "sssp, 600 K vertices", "kind": "sssp", "n": 600_013, "ef": 16},
        # The largest one: 0.27 G CSR entries.
        {"name": "sssp, 8.4 M vertices", "kind": "sssp", "n": 1 << 23, "ef": 16},
        # The benchmark's edge list, a range that is no multiple of anything.
        {"name": "generate, 50 M edges", "kind": "generate", "scale": 22, "start": 1_000_003, "count": 50_000_021},
        # Graph construction from an edge list the user has.
        {"name": "build, 3 M vertices", "kind": "build", "n": 3_000_017, "ef": 16},
        # The benchmark's whole protocol for one root.
        {"name": "runner, 1 M vertices", "kind": "runner", "n": 1 << 20, "ef": 16},
        # A full batch of searches on the graph of the benchmark's middle scale.
        {"name": "msbfs, 256 x 4.2 M vertices", "kind": "msbfs", "n": 1 << 22, "ef": 16, "roots": 256},
        # Batched shortest paths, as a server of many small queries runs them.
        {"name": "sssp multi, 32 x 130 K", "kind": "sssp_multi", "n": 1 << 17, "ef": 16, "roots": 32},
        # Many small graphs of SCALE 10 to 18 in one captured batch.
        {"name": "packed, 90 graphs", "kind": "packed", "graphs": 90, "lo": 10, "hi": 18, "ef": 16},
    ]


def _between(rng, lo, hi):
    """A whole number, even over the logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["bfs_query", "bfs", "sssp", "generate", "build", "runner", "msbfs", "sssp_multi", "packed"])
    c = {"kind": kind}
    if kind == "generate":
        c["scale"] = rng.randint(10, 26)
        c["count"] = _between(rng, 1 << 10, min(50_000_000, 16 << c["scale"]))
        c["start"] = rng.randint(0, (16 << c["scale"]) - c["count"])
        return c
    if kind == "packed":
        c["lo"] = rng.randint(8, 12)
        c["hi"] = rng.randint(c["lo"], 16)
        c["graphs"] = _between(rng, 4, 90)
        c["ef"] = rng.choice([8, 16])
        return c
    top = {"bfs_query": 1 << 20, "bfs": 1 << 25, "sssp": 1 << 23, "build": 3_000_000, "runner": 1 << 20,
           "msbfs": 1 << 22, "sssp_multi": 1 << 17}[kind]
    c["n"] = _between(rng, 1 << 11, top)
    c["ef"] = rng.choice([8, 16, 16, 32]) if c["n"] <= top // 2 else rng.choice([8, 16])
    if kind == "msbfs":
        c["roots"] = rng.randint(8, 256)
    if kind == "sssp_multi":
        c["roots"] = rng.randint(2, 32)
    return c


# ----------------------------------------------------------------- inputs ----

CHUNK = 1 << 25  # edges generated at a time
LOOPS = 1009  # one edge of so many is a self-loop, so that every seed's graph has as many entries


def _edges(n, ef, seed):
    """(int64[n * ef, 2] edges, float32 weights) of a Kronecker graph of n vertices."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    scale = max(1, (n - 1).bit_length())
    m = n * ef
    name = torch.randperm(1 << scale, generator=gen, device=DEV) % n
    edges = torch.empty((m, 2), dtype=torch.int64, device=DEV)
    for lo in range(0, m, CHUNK):
        k = min(CHUNK, m - lo)
        u = torch.zeros(k, dtype=torch.int32, device=DEV)
        v = torch.zeros(k, dtype=torch.int32, device=DEV)
        for _ in range(scale):
            r = torch.rand(k, generator=gen, device=DEV)
            down = r >= 0.76
            right = ((r >= 0.57) & ~down) | (r >= 0.95)
            u = (u << 1) + down
            v = (v << 1) + right
        u, v = name[u.long()], name[v.long()]
        v = torch.where(u == v, (u + 1) % n, v)
        edges[lo:lo + k, 0], edges[lo:lo + k, 1] = u, v
    edges[::LOOPS, 1] = edges[::LOOPS, 0]
    return edges, torch.rand(m, generator=gen, device=DEV)


def _roots(edges, n, count, seed):
    """`count` vertices within two hops of the highest-degree vertex."""
    gen = torch.Generator(device=DEV).manual_seed(seed + 1)
    near = torch.zeros(n, dtype=torch.bool, device=DEV)
    near[torch.argmax(torch.bincount(edges[:, 0], minlength=n))] = True
    for _ in range(2):
        for a, b in ((0, 1), (1, 0)):
            near[edges[:, b][near[edges[:, a]]]] = True
    near = near.nonzero()[:, 0]
    return near[torch.randperm(near.numel(), generator=gen, device=DEV)[:count]].tolist()


def _graph(edges, weights, n, **options):
    return G.oned_graph_from_tuple_graph(G.TupleGraph(edges, weights, edges.shape[0]), n, **options)


def _packed_sizes(case):
    """Scales lo..hi in turn."""
    return [case["lo"] + i % (case["hi"] - case["lo"] + 1) for i in range(case["graphs"])]


def _packed_inputs(case, seed):
    for i, scale in enumerate(_packed_sizes(case)):
        edges, weights = _edges(1 << scale, case["ef"], seed * 1009 + i)
        yield 1 << scale, edges, weights, _roots(edges, 1 << scale, 1, seed * 1009 + i)[0]


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "generate":
        s["seed"] = G.make_mrg_seed(seed, 3)
        s["scale"], s["start"], s["end"] = case["scale"], case["start"], case["start"] + case["count"]
        m = case["count"]
        s["out"] = G.TupleGraph(torch.empty((m, 2), dtype=torch.int64, device=DEV),
                                torch.empty(m, dtype=torch.float32, device=DEV), m)
        return s
    if kind == "packed":
        graphs, roots = [], []
        for n, edges, weights, root in _packed_inputs(case, seed):
            graphs.append(_graph(edges, weights, n, bfs_order=False, sssp_renumber=False, with_main=False))
            roots.append(root)
        s["batch"] = G.PackedBatch(G.pack_graphs(graphs, roots))
        return s
    n = s["n"] = case["n"]
    edges, weights = _edges(n, case["ef"], seed)
    if kind == "build":
        s["edges"], s["weights"] = edges, weights
        return s
    s["roots"] = _roots(edges, n, case.get("roots", 1), seed)
    searches_only = kind in ("bfs", "bfs_query", "msbfs")  # a program without shortest paths skips their copy
    g = s["graph"] = _graph(edges, weights, n, sssp_renumber=not searches_only)
    del edges, weights
    if kind in ("bfs", "bfs_query", "runner"):
        s["bfs"] = G.BfsState(g)
    if kind in ("sssp", "runner"):
        s["sssp"] = G.SsspState(g)
    if kind == "msbfs":
        s["ms"] = G.MsBfsState(g)
        s["bytes"] = torch.empty((len(s["roots"]), n), dtype=torch.uint8, device=DEV)
    if kind == "sssp_multi":
        s["work"] = G.sssp_multi_workspace(g)
        s["dist"] = torch.empty((len(s["roots"]), n), dtype=torch.float32, device=DEV)
        s["pred"] = torch.empty((len(s["roots"]), n), dtype=torch.int64, device=DEV)
    return s


# -------------------------------------------------------------------- run ----

def run(s):
    kind = s["kind"]
    if kind == "generate":
        t = G.generate_kronecker_range(s["seed"], s["scale"], s["start"], s["end"], out=s["out"])
        return {"edges": t.edges, "weights": t.weights}
    if kind == "packed":
        b = s["batch"]
        b.run()
        return {"depth": b.bfs.depth, "dist": b.sssp.dist, "pred": b.sssp.pred}
    if kind == "build":
        g = _graph(s["edges"], s["weights"], s["n"])
        r = g.sr
        return {"rowstarts": g.rowstarts, "col": g.col, "w": g.w, "scol": g.scol, "sw": g.sw, "light": g.light_deg,
                "tiny": g.tiny_deg, "bcol": g.bcol, "btop": g.btop, "isolated": g.isolated,
                "main": g.main_bits.view(np.int32), "r_rowstarts": r.rowstarts, "r_col": r.col, "r_w": r.w,
                "r_light": r.light_deg, "r_tiny": r.tiny_deg, "perm": r.perm, "inv": r.inv}
    g, root = s["graph"], s["roots"][0]
    if kind == "bfs_query":
        G.oned_graph_bfs_reset(s["bfs"], True, g)
        st = G.oned_graph_bfs_query(g, s["bfs"], root, with_depth=True)
        return {"depth": s["bfs"].depth, "reached": int(st.reached)}
    if kind == "bfs":
        G.oned_graph_bfs_run(g, s["bfs"], root)
        return {"depth": s["bfs"].depth}
    if kind == "sssp":
        G.oned_graph_sssp_run(g, s["sssp"], root)
        return {"dist": s["sssp"].dist, "pred": s["sssp"].pred}
    if kind == "msbfs":
        G.msbfs_run(g, s["ms"], s["roots"], sync=False)
        return {"depths": G.msbfs_depths_u8(s["ms"], out=s["bytes"])}
    if kind == "sssp_multi":
        G.oned_graph_sssp_multi(g, s["roots"], work=s["work"], dist=s["dist"], pred=s["pred"], sync=False)
        return {"dist": s["dist"], "pred": s["pred"]}
    if kind == "runner":
        bfs, sssp = s["bfs"], s["sssp"]
        G.oned_graph_bfs_reset(bfs, True, g)
        G.oned_graph_bfs_traverse(g, bfs, root)
        hops = G.bfs_compute_dist_from_pred(g, bfs, root)
        bad = G.bfs_validate(g, root, bfs.pred, hops, work=bfs.val_work)
        edges = G.edge_count(g, bfs.pred, work=bfs.val_work)
        G.oned_graph_sssp_reset(sssp)
        G.oned_graph_sssp_traverse(g, sssp, root)
        worse = G.sssp_validate(g, root, sssp.dist, sssp.pred, work=bfs.val_work)
        return {"depth": bfs.depth, "hops": hops, "bfs_errors": bad, "edges": edges, "dist": sssp.dist,
                "pred": sssp.pred, "sssp_errors": worse}
    raise ValueError(f"unknown kind {kind!r}")


# ------------------------------------------------------------------- work ----

def work(case):
    """Inputs read once and outputs written once; no floating-point work to speak of."""
    kind = case["kind"]
    if kind == "generate":
        return {"bytes": 20 * case["count"], "flops": 0}
    if kind == "packed":
        n = sum(1 << s for s in _packed_sizes(case))
    else:
        n = case["n"]
    e = 2 * case["ef"] * n  # CSR entries, self-loops aside
    bfs = 4 * e + 8 * n + 12 * n   # column, row starts; parents and depths
    sssp = 8 * e + 8 * n + 12 * n  # column, weights, row starts; distances and parents
    if kind in ("bfs", "bfs_query"):
        b = bfs
    elif kind == "sssp":
        b = sssp
    elif kind == "packed":
        b = bfs + sssp
    elif kind == "msbfs":
        b = 4 * e + 8 * n + case["roots"] * n
    elif kind == "sssp_multi":
        b = 8 * e + 8 * n + case["roots"] * 12 * n
    elif kind == "build":  # edge list in; three copies of the column and weights, the BFS's column and the vertex arrays out
        b = 10 * e + 8 * e * 3 + 4 * e + 44 * n
    else:  # runner: the searches, the distances, the two validations and the edge count each read the graph
        b = bfs + sssp + (4 * e + 24 * n) + (4 * e + 24 * n) + (4 * e + 16 * n) + (8 * e + 20 * n)
    return {"bytes": b, "flops": 0}


# ------------------------------------------------------------------ exact ----

def _shortest(edges, weights, n, roots):
    """float64[n] distances from the nearest root, -1 where unreached: every
    edge of the vertices that came nearer relaxed, until none does."""
    # Non-negative doubles order like their bits, which have a fast atomic minimum.
    top = torch.iinfo(torch.int64).max
    dist = torch.full((n,), top, dtype=torch.int64, device=DEV)
    dist[torch.as_tensor(roots, device=DEV)] = 0
    moved = dist == 0
    while bool(moved.any()):
        old = dist.clone()
        for lo in range(0, edges.shape[0], CHUNK):
            e, w = edges[lo:lo + CHUNK], weights[lo:lo + CHUNK]
            for a, b in ((0, 1), (1, 0)):
                live = moved[e[:, a]]
                u, v = e[:, a][live], e[:, b][live]
                cand = (old[u].view(torch.float64) + w[live].double()).view(torch.int64)
                dist.scatter_reduce_(0, v, cand, "amin")
        moved = dist != old
    far = dist == top
    out = dist.view(torch.float64).clone()
    out[far] = -1.0
    return out


def _built_weights(edges, weights, n, light=0.1, tiny=0.1 / 30):
    """The weights in the canonical order, the split copy's and the renumbered copy's."""
    keep = edges[:, 0] != edges[:, 1]
    u, v, w = edges[keep, 0], edges[keep, 1], weights[keep]
    src, dst, w = torch.cat([u, v]), torch.cat([v, u]), torch.cat([w, w])
    order = torch.argsort(w, stable=True)
    order = order[torch.argsort((src * n + dst)[order], stable=True)]
    src, w = src[order], w[order]
    part = (w >= np.float32(tiny)).long() + (w >= np.float32(light)).long()
    order = torch.argsort(src * 4 + part, stable=True)
    degree = torch.bincount(src, minlength=n)
    perm = torch.empty(n, dtype=torch.int64, device=DEV)
    perm[torch.argsort(-degree, stable=True)] = torch.arange(n, device=DEV)
    split = w[order]
    renumbered = split[torch.argsort(perm[src[order]], stable=True)]
    return w.double(), split.double(), renumbered.double()


def exact(case, seed):
    kind = case["kind"]
    if kind == "packed":
        parts = [_shortest(edges, weights, n, [root]) for n, edges, weights, root in _packed_inputs(case, seed)]
        return {"depth": None, "dist": torch.cat(parts), "pred": None}
    if kind not in ("sssp", "sssp_multi", "runner", "build"):
        return None
    n = case["n"]
    edges, weights = _edges(n, case["ef"], seed)
    if kind == "build":
        w, sw, r_w = _built_weights(edges, weights, n)
        names = ("rowstarts", "col", "scol", "light", "tiny", "bcol", "btop", "isolated", "main", "r_rowstarts",
                 "r_col", "r_light", "r_tiny", "perm", "inv")
        return {**dict.fromkeys(names), "w": w, "sw": sw, "r_w": r_w}
    roots = _roots(edges, n, case.get("roots", 1), seed)
    if kind == "sssp_multi":
        return {"dist": torch.stack([_shortest(edges, weights, n, [r]) for r in roots]), "pred": None}
    out = {"dist": _shortest(edges, weights, n, roots[:1]), "pred": None}
    if kind == "runner":
        out |= dict.fromkeys(("depth", "hops", "bfs_errors", "edges", "sssp_errors"))
    return out
