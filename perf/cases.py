"""Performance cases: what users of enterprise_b200 have it do, through its public entry points.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare`` makes what
a program holds before the call (device graphs, sources, output buffers, plans, a server), ``run``
makes one call, and ``work`` states what the call cannot do without: the CSR read once (8-byte
offsets, 4-byte neighbours) and each output written once. A breadth-first search does no floating-point
work, and its depths are whole numbers, so ``exact`` has nothing to give.

Graphs are the repository's own seeded generators (R-MAT with the Graph500 parameters, Erdos-Renyi,
2D grids with 10% of the edges dropped); every input follows from the seed. Kinds of calls:

  host     Graph.bfs: one source, depths in a fresh host array
  single   Graph.bfs_device: one source, depths stay on the GPU
  many     Graph.bfs_many: a list of sources, each row copied to a page-locked host array of bytes
  certify  Graph.bfs_device with parents, then Graph.validate_device of both
  batch    Graph.bfs_batch_device(_u8): many sources at once, rows on the GPU
  multi    MultiPlan.run and .depths: many graphs of uneven sizes, each with its own sources
  serve    Server: a burst of queries on resident graphs, their depths read back
  noalloc  ent_bfs_noalloc: a caller's CSR, no allocation
  build    Graph.from_edges of a host edge list, one traversal, the CSR read back
"""
import ctypes
import math

import numpy as np
import torch

import enterprise_b200 as eb
from enterprise_b200 import tune


def listed():
    return [
        # A small graph queried from a script: the call's latency and launches are all there is.
        {"name": "host_rmat12", "kind": "host", "graph": "rmat", "scale": 12, "degree": 16},
        # An ordinary graph with the options as they come, depths used on the GPU.
        {"name": "single_rmat20", "kind": "single", "graph": "rmat", "scale": 20, "degree": 16, "tuned": False},
        # The headline workload: one source on R-MAT scale 24, edge factor 16, with the options shipped for it.
        {"name": "single_rmat24", "kind": "single", "graph": "rmat", "scale": 24, "degree": 16, "tuned": True},
        # A road-like graph: thousands of levels of small frontiers.
        {"name": "single_grid4096", "kind": "single", "graph": "grid", "width": 4096, "height": 4096, "tuned": False},
        # The reference's own loop on the headline graph: a list of sources, each one's byte depths to the host.
        {"name": "many_rmat24", "kind": "many", "graph": "rmat", "scale": 24, "degree": 16, "tuned": True, "sources": 16},
        # What enterprise.bin does by default: traverse, then certify every vertex and edge; a uniform graph of odd size.
        {"name": "certify_er4m", "kind": "certify", "graph": "er", "vertices": 4194301, "degree": 16},
        # The batched headline: 256 sources, int32 rows.
        {"name": "batch256_rmat22", "kind": "batch", "graph": "rmat", "scale": 22, "degree": 16, "sources": 256, "bytes": False},
        # All-pairs style statistics on a mid-sized graph: a wide, ragged batch with byte rows.
        {"name": "batch1000_rmat20", "kind": "batch", "graph": "rmat", "scale": 20, "degree": 16, "sources": 1000, "bytes": True},
        # A dataset of graphs of uneven sizes, each with its own number of sources.
        {"name": "multi24", "kind": "multi", "graphs": 24, "low": 12, "high": 18, "most": 64},
        # A burst of queries against resident graphs, shallow ones and a deep one.
        {"name": "serve48", "kind": "serve", "queries": 48, "low": 14, "high": 18, "side": 512},
        # A caller that may not allocate, on a mid-sized graph.
        {"name": "noalloc_rmat18", "kind": "noalloc", "graph": "rmat", "scale": 18, "degree": 16},
        # A one-off: a raw edge list (repeats and loops in it) to a resident graph, one traversal, the CSR saved.
        {"name": "build_rmat18", "kind": "build", "scale": 18, "edges": 4194304},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _graph(rng, kinds, low, high):
    """A graph of about 2^low to 2^high vertices, and its description."""
    kind = rng.choice(kinds)
    if kind == "rmat":
        return {"graph": "rmat", "scale": rng.randint(low, high), "degree": rng.randint(8, 32)}
    n = _log(rng, 1 << low, 1 << high)
    if kind == "er":
        return {"graph": "er", "vertices": n | 1, "degree": rng.randint(6, 32)}
    w = max(2, int(math.sqrt(n) * rng.uniform(0.5, 1.5)))
    return {"graph": "grid", "width": w, "height": max(2, n // w)}


def draw(rng):
    kind = rng.choice(["host", "single", "single", "many", "certify", "batch", "batch", "multi", "serve", "noalloc", "build"])
    case = {"kind": kind}
    if kind == "host":
        case.update(_graph(rng, ["rmat", "rmat", "er"], 10, 20))
    elif kind == "single":
        case.update(_graph(rng, ["rmat", "rmat", "er", "grid"], 14, 22), tuned=False)
    elif kind == "many":
        case.update(_graph(rng, ["rmat", "rmat", "er"], 18, 22), tuned=False, sources=rng.randint(5, 48))
    elif kind == "certify":
        case.update(_graph(rng, ["rmat", "er"], 16, 22))
    elif kind == "batch":
        case.update(_graph(rng, ["rmat", "rmat", "rmat", "er", "grid"], 14, 20), bytes=rng.random() < 0.5)
        if case["graph"] == "grid":
            case.update(sources=rng.randint(3, 32), bytes=False)  # depths above 254
        else:
            case.update(sources=_log(rng, 3, 1024))
    elif kind == "multi":
        low = rng.randint(10, 13)
        case.update(graphs=rng.randint(5, 40), low=low, high=low + rng.randint(1, 5), most=_log(rng, 4, 100))
    elif kind == "serve":
        low = rng.randint(11, 15)
        case.update(queries=rng.randint(9, 60), low=low, high=low + rng.randint(1, 4), side=rng.randint(100, 700))
    elif kind == "noalloc":
        case.update(_graph(rng, ["rmat", "rmat", "er", "grid"], 10, 19))
    else:
        scale = rng.randint(12, 20)
        case.update(scale=scale, edges=_log(rng, 1 << scale, 1 << (scale + 4)) | 1)
    return case


# ---------------------------------------------------------------- inputs ----

def _make(case, seed):
    if case["graph"] == "rmat":
        return eb.Graph.rmat(case["scale"], case["degree"], seed=seed)
    if case["graph"] == "er":
        return eb.Graph.er(case["vertices"], case["degree"], seed=seed)
    return eb.Graph.grid(case["width"], case["height"], 0.1, seed=seed)


class _DeviceArray:
    def __init__(self, ptr, n, kind):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": kind, "version": 2}


def _sources(g, n, seed):
    """n seeded non-isolated vertices (the reference's rule for its sources)."""
    off = torch.as_tensor(_DeviceArray(g.device_csr()[0], g.vert_count + 1, "<i8"), device="cuda")
    some = torch.nonzero(off[1:] > off[:-1]).flatten()
    at = torch.from_numpy(np.random.RandomState(seed % (1 << 31)).randint(0, max(1, some.numel()), n))
    return some[at.to(some.device)].cpu().numpy().astype(np.int32)


def _options(g, case):
    """The options shipped with the package for this graph class, where it ships any."""
    if case.get("tuned"):
        key = tune.TuneCache.key(tune.gpu_name(), tune.graph_class(g.vert_count, g.edge_count, "rmat"), "single")
        best = tune.TuneCache().get(key)
        if best is not None:
            g.opts = best


def _edges(scale, n, seed):
    """A raw edge list as a crawler or converter leaves it: R-MAT draws with repeats and loops, host int64."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.zeros(n, dtype=torch.int64, device="cuda")
    v = torch.zeros(n, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(n, device="cuda", generator=gen)
        u = 2 * u + (r >= 0.76)
        v = 2 * v + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    ids = torch.randperm(1 << scale, device="cuda", generator=gen)
    return ids[u].cpu().numpy(), ids[v].cpu().numpy()


def _scales(case, n):
    return [case["low"] + (k * (case["high"] - case["low"])) // max(1, n - 1) for k in range(n)]


def _counts(case):
    """Sources of each graph of a multi case: uneven, 1 to case["most"], the case's own."""
    return np.random.RandomState(case["graphs"]).randint(1, case["most"] + 1, case["graphs"])


_streams = {}


def _stream():
    """The one stream on which a program does its GPU work."""
    if "own" not in _streams:
        _streams["own"] = torch.cuda.Stream()
    return _streams["own"].cuda_stream


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.RandomState(seed % (1 << 31))
    state = {"kind": kind}
    if kind == "build":
        src, dst = _edges(case["scale"], case["edges"], seed)
        n = 1 << case["scale"]
        # the program's own arrays for the CSR: an undirected edge list has at most two entries an edge
        state.update(src=src, dst=dst, n=n, source=int(src[rng.randint(len(src))]),
                     beg_pos=np.zeros(n + 1, dtype=np.int64), csr=np.full(2 * len(src), -1, dtype=np.int32))
        return state
    if kind == "multi":
        graphs = [eb.Graph.rmat(s, int(rng.randint(8, 33)), seed=seed + 977 * k)
                  for k, s in enumerate(_scales(case, case["graphs"]))]
        lists = [_sources(g, int(n), seed + k) for k, (g, n) in enumerate(zip(graphs, _counts(case)))]
        state.update(plan=eb.MultiPlan(graphs, lists), n=len(graphs))
        return state
    if kind == "serve":
        graphs = [eb.Graph.rmat(s, 16, seed=seed + 977 * k) for k, s in enumerate(_scales(case, 3))]
        graphs.append(eb.Graph.grid(case["side"], case["side"], 0.1, seed=seed))
        which = np.random.RandomState(case["queries"]).randint(0, len(graphs), case["queries"])
        picks = [_sources(g, case["queries"], seed + k) for k, g in enumerate(graphs)]
        state.update(server=eb.Server(graphs, rows_per_graph=case["queries"]),
                     queries=[(int(k), int(picks[k][i])) for i, k in enumerate(which)])
        return state
    g = _make(case, seed)
    V = g.vert_count
    state.update(g=g, stream=_stream())
    if kind in ("host", "single", "certify", "noalloc"):
        state.update(source=int(_sources(g, 1, seed)[0]))
        state.update(depth=torch.empty(V, dtype=torch.int32, device="cuda") if kind != "host" else None)
        state.update(parent=torch.empty(V, dtype=torch.int32, device="cuda") if kind == "certify" else None)
        _options(g, case)
        if kind == "noalloc":
            f = eb.lib().ent_bfs_noalloc
            f.restype = ctypes.c_int
            f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p]
            state.update(call=f, csr=g.device_csr())
    elif kind == "many":
        state.update(sources=_sources(g, case["sources"], seed))
        state.update(rows=torch.empty((case["sources"], V), dtype=torch.uint8, pin_memory=True).numpy())
        _options(g, case)
    else:
        n = case["sources"]
        state.update(sources=_sources(g, n, seed), bytes=case["bytes"],
                     rows=torch.empty((n, V), dtype=torch.uint8 if case["bytes"] else torch.int32, device="cuda"))
    return state


# ------------------------------------------------------------------ runs ----

def _serve(server, queries):
    ids = [server.submit(k, s) for k, s in queries]
    open_ids, rows = set(ids), {}
    while open_ids:
        for r in server.poll(wait_us=1000):
            q = r["query_id"]
            if r["status"] != 0:
                raise RuntimeError("query %d ended with status %d" % (q, r["status"]))
            rows[q] = server.depth(q)
            server.release(q)
            open_ids.discard(q)
    return [rows[q] for q in ids]


def run(state):
    kind = state["kind"]
    if kind == "host":
        return state["g"].bfs(state["source"])[0]
    if kind == "single":
        state["g"].bfs_device(state["source"], state["depth"].data_ptr(), stream=state["stream"], stats=False)
        return state["depth"]
    if kind == "many":
        state["g"].bfs_many(state["sources"], list(state["rows"]))
        return state["rows"]
    if kind == "certify":
        # parents are any of a vertex's valid ones: the certificate answers for them
        g, d, p = state["g"], state["depth"], state["parent"]
        g.bfs_device(state["source"], d.data_ptr(), p.data_ptr())
        certificate = g.validate_device(state["source"], d.data_ptr(), p.data_ptr())
        return {"depth": d, "certificate": certificate}
    if kind == "batch":
        call = state["g"].bfs_batch_device_u8 if state["bytes"] else state["g"].bfs_batch_device
        call(state["sources"], state["rows"].data_ptr(), stream=state["stream"], stats=False)
        return state["rows"]
    if kind == "multi":
        state["plan"].run()
        return [state["plan"].depths(k) for k in range(state["n"])]
    if kind == "serve":
        return _serve(state["server"], state["queries"])
    if kind == "noalloc":
        beg, adj = state["csr"]
        status = state["call"](beg, adj, state["g"].vert_count, state["source"], state["depth"].data_ptr(), None)
        if status != 0:
            raise RuntimeError("ent_bfs_noalloc: status %d" % status)
        return state["depth"]
    with eb.Graph.from_edges(state["src"], state["dst"], state["n"]) as g:
        depth = g.bfs(state["source"])[0]
        status = eb.lib().ent_graph_download(g.handle, state["beg_pos"].ctypes.data_as(ctypes.POINTER(ctypes.c_int64)),
                                             state["csr"].ctypes.data_as(ctypes.POINTER(ctypes.c_int32)))
        if status != 0:
            raise RuntimeError("ent_graph_download: status %d" % status)
    return {"beg_pos": state["beg_pos"], "csr": state["csr"], "depth": depth}


# ------------------------------------------------------------------ work ----

def _size(case):
    """Vertices and directed CSR entries (about: repeats and loops that the generators drop are counted)."""
    if case["graph"] == "rmat":
        return 1 << case["scale"], 2 * case["degree"] << case["scale"]
    if case["graph"] == "er":
        return case["vertices"], case["vertices"] * case["degree"]
    n = case["width"] * case["height"]
    return n, int(3.6 * n)


def work(case):
    kind = case["kind"]
    if kind == "multi":
        b = sum((8 + 160 + 4 * int(n)) << s for s, n in zip(_scales(case, case["graphs"]), _counts(case)))
    elif kind == "serve":
        sizes = [(1 << s, 32 << s) for s in _scales(case, 3)] + [(case["side"] ** 2, int(3.6 * case["side"] ** 2))]
        b = sum(8 * v + 4 * e + 4 * v * case["queries"] / 4 for v, e in sizes)
    elif kind == "build":
        v, e = 1 << case["scale"], 2 * case["edges"]
        b = 16 * case["edges"] + 8 * v + 4 * e + 4 * v  # edge list in, CSR and depths out
    else:
        v, e = _size(case)
        reads = case["sources"] if kind == "many" else 2 if kind == "certify" else 1  # traversals, and the check's own read
        row = 1 if kind == "many" or case.get("bytes") else 8 if kind == "certify" else 4
        b = reads * (8 * v + 4 * e) + row * v * case.get("sources", 1)
    return {"bytes": float(b), "flops": 0.0}


def exact(case, seed):
    return None
