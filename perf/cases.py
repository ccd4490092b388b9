"""The work that programs have this library do, as measurable cases.

A case is a dict of plain values.  Its "kind" is the call that is measured:

  flow      a new edge list through the whole path, as one run of the C driver
            does it: sort + CSR (both directions), one direction-optimized BFS
            and a PageRank pull of 20 iterations (the driver's default)
  build     sort + CSR of both directions from device edge arrays
  bfs       one direction-optimized search on a resident graph
  dropin    the same search through the C API's breadthFirstSearchGraphCSR on
            a host GraphCSR, results in host arrays
  pagerank  20 iterations on a resident graph, pull (mode 0) or push (mode 1)
  spmv      20 SPMV passes on a resident graph, pull (mode 0) or push (mode 1)
  msbfs     64 searches at once, a bit-lane per root
  ppr       10 iterations of personalized PageRank for 32 seeds
  batch     many small graphs at once: a BFS of each and 20 PageRank iterations

"graph" is "rmat" (a/b/c/d = .57/.19/.19/.05, ids permuted, V = 2^scale),
"uniform" (V vertices, uniform ids) or "grid" (V = side^2, four neighbours,
both directions, and a diagonal shortcut per vertex with probability 1e-4).
Self loops and duplicate edges are kept.  "E" is the number of edges (a grid's
follows from its side).  "weighted": float32 weights in [1, 256).  "sort" is
SORT_TYPE: 0 by source, 1 by source and destination.

Depths, counts, CSR arrays and ranks are returned.  The parents of a search
are not: which frontier vertex claims a vertex top-down is a race, in the
library as in the C code it replaces, so two runs differ in them.
"""
import ctypes
import os
import tempfile

import numpy as np
import torch

import opengraph_b200 as og

DAMP = float(np.float32(0.85))
BASE = float(np.float32(1.0) - np.float32(0.85))


def listed():
    return [
        # a whole run on a small new edge list (RMAT-16): what a program pays
        # when nothing of the graph is prepared; launches and waits count most
        {"name": "flow_rmat16", "kind": "flow", "graph": "rmat", "scale": 16, "E": 1048573, "weighted": False,
         "sort": 0, "iters": 20},
        # the preparation of the headline graph, weighted
        {"name": "build_rmat22_w", "kind": "build", "graph": "rmat", "scale": 22, "E": 67108864, "weighted": True,
         "sort": 0},
        # the other sort type, no hubs, sizes that are no multiple of anything
        {"name": "build_uniform_lex", "kind": "build", "graph": "uniform", "V": 1500007, "E": 20000003,
         "weighted": False, "sort": 1},
        # the smallest call: a C program's search of a small host graph
        {"name": "dropin_rmat14", "kind": "dropin", "graph": "rmat", "scale": 14, "E": 262144, "sort": 0},
        # the headline search
        {"name": "bfs_rmat22", "kind": "bfs", "graph": "rmat", "scale": 22, "E": 67108864, "weighted": False,
         "sort": 0},
        # a high-diameter search: about two thousand small steps
        {"name": "bfs_grid1000", "kind": "bfs", "graph": "grid", "side": 1000, "weighted": False, "sort": 0},
        # PageRank of the headline graph
        {"name": "pagerank_pull_rmat22", "kind": "pagerank", "graph": "rmat", "scale": 22, "E": 67108864,
         "weighted": False, "sort": 0, "mode": 0, "iters": 20},
        # the push form on an ordinary graph of odd size
        {"name": "pagerank_push_rmat20", "kind": "pagerank", "graph": "rmat", "scale": 20, "E": 20971519,
         "weighted": False, "sort": 0, "mode": 1, "iters": 20},
        # weighted SPMV of an ordinary graph
        {"name": "spmv_pull_rmat20_w", "kind": "spmv", "graph": "rmat", "scale": 20, "E": 16777216,
         "weighted": True, "sort": 0, "mode": 0, "iters": 20},
        # batched searches (all-pairs samples, landmarks)
        {"name": "msbfs_rmat20", "kind": "msbfs", "graph": "rmat", "scale": 20, "E": 16777216, "roots": 64},
        # batched personalized PageRank (recommendation seeds)
        {"name": "ppr_rmat20", "kind": "ppr", "graph": "rmat", "scale": 20, "E": 16777216, "seeds": 32, "iters": 10},
        # many uneven small graphs (scales 10 to 15, edge factors 8 to 32)
        {"name": "batch_rmat10_15", "kind": "batch", "graphs": 96, "lo": 10, "hi": 15, "ef_lo": 8, "ef_hi": 32,
         "iters": 20},
    ]


def draw(rng):
    kind = rng.choice(["flow", "build", "build", "dropin", "bfs", "bfs", "pagerank", "pagerank", "spmv", "msbfs", "ppr",
                       "batch"])
    if kind == "batch":
        lo = rng.randint(8, 11)
        return {"kind": kind, "graphs": rng.randint(3, 128), "lo": lo, "hi": rng.randint(lo, 15), "ef_lo": 8,
                "ef_hi": rng.randint(8, 32), "iters": rng.randint(5, 30)}
    top = {"flow": 22, "build": 22, "dropin": 20, "bfs": 22, "pagerank": 22, "spmv": 22, "msbfs": 21, "ppr": 21}[kind]
    scale = rng.uniform(12.0, top)
    c = {"kind": kind}
    how = rng.random()
    if kind == "bfs" and how < 0.25:
        c.update(graph="grid", side=int(2.0 ** rng.uniform(5.0, 10.0)))
    elif how < 0.65:
        c.update(graph="rmat", scale=int(round(scale)))
    else:
        c.update(graph="uniform", V=int(2.0 ** scale) | 1)
    if c["graph"] != "grid":
        V = 1 << c["scale"] if c["graph"] == "rmat" else c["V"]
        c["E"] = min(67108864, int(V * rng.uniform(4.0, 32.0)))
        if kind in ("msbfs", "ppr"):
            c["E"] = min(33554432, c["E"])
    c["sort"] = rng.choice([0, 0, 1])
    if kind in ("flow", "build", "bfs", "pagerank", "spmv"):
        c["weighted"] = rng.random() < 0.5
    if kind in ("pagerank", "spmv"):
        c["mode"] = rng.randint(0, 1)
    if kind in ("flow", "pagerank", "spmv"):
        c["iters"] = rng.randint(5, 20)
    if kind == "msbfs":
        c["roots"] = rng.randint(3, 64)
    if kind == "ppr":
        c.update(seeds=rng.randint(1, 32), iters=rng.randint(2, 10))
    return c


# ------------------------------------------------------------------ inputs --

def _vertices(case):
    if case["graph"] == "rmat":
        return 1 << case["scale"]
    return case["side"] ** 2 if case["graph"] == "grid" else case["V"]


def _rmat(scale, E, gen):
    """RMAT ids of a 2^scale-vertex graph, permuted (device int32)."""
    src = torch.zeros(E, dtype=torch.int32, device="cuda")
    dst = torch.zeros(E, dtype=torch.int32, device="cuda")
    for _ in range(scale):
        u = torch.rand(E, generator=gen, device="cuda")
        down = u >= 0.76
        src.mul_(2).add_(down)
        dst.mul_(2).add_(((u >= 0.57) & ~down) | (u >= 0.95))
    perm = torch.randperm(1 << scale, generator=gen, device="cuda", dtype=torch.int32)
    return perm[src], perm[dst]


def _grid(side, gen):
    ids = torch.arange(side * side, dtype=torch.int32, device="cuda").view(side, side)
    pairs = [(ids[:, :-1].reshape(-1), ids[:, 1:].reshape(-1)), (ids[:-1].reshape(-1), ids[1:].reshape(-1))]
    jump = torch.rand(side - 1, side - 1, generator=gen, device="cuda") < 1e-4
    pairs.append((ids[:-1, :-1][jump], ids[1:, 1:][jump]))
    a = torch.cat([p[0] for p in pairs])
    b = torch.cat([p[1] for p in pairs])
    src, dst = torch.cat([a, b]), torch.cat([b, a])
    order = torch.randperm(src.numel(), generator=gen, device="cuda")
    return src[order].contiguous(), dst[order].contiguous()


def _edges(case, seed):
    """(V, src, dst, weight or None) on the device, and the generator."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000003 * int(seed) + 17)
    V = _vertices(case)
    if case["graph"] == "rmat":
        src, dst = _rmat(case["scale"], case["E"], gen)
    elif case["graph"] == "grid":
        src, dst = _grid(case["side"], gen)
    else:
        src = torch.randint(0, V, (case["E"],), generator=gen, device="cuda", dtype=torch.int32)
        dst = torch.randint(0, V, (case["E"],), generator=gen, device="cuda", dtype=torch.int32)
    w = None
    if case.get("weighted"):
        w = torch.rand(src.numel(), generator=gen, device="cuda").mul_(255.0).add_(1.0)
    return V, src, dst, w, gen


def _roots(src, V, n, gen):
    """n distinct vertices with out-edges, drawn from the seed."""
    cand = torch.unique(src)
    pick = torch.randperm(cand.numel(), generator=gen, device="cuda")[:n]
    return [int(x) for x in cand[pick].tolist()]


def _batch_edges(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000003 * int(seed) + 29)
    rng = np.random.default_rng(case["graphs"])  # the graphs' sizes belong to the case
    nv, off, ss, dd, roots = [], [0], [], [], []
    for _ in range(case["graphs"]):
        scale = int(rng.integers(case["lo"], case["hi"] + 1))
        E = int((1 << scale) * rng.integers(case["ef_lo"], case["ef_hi"] + 1)) - int(rng.integers(0, 5))
        s, d = _rmat(scale, E, gen)
        nv.append(1 << scale)
        off.append(off[-1] + E)
        ss.append(s)
        dd.append(d)
        roots.append(int(s[0]))
    return nv, off, torch.cat(ss), torch.cat(dd), roots


class _HostGraph:
    """A host GraphCSR made by the C API from an edge file, freed with it."""

    def __init__(self, src, dst, sort):
        self.lib = og.load(False)
        self.lib.quiet(True)
        fd, path = tempfile.mkstemp(suffix=".bin")
        os.close(fd)
        try:
            og.write_edge_file(path, src.cpu().numpy().view(np.uint32), dst.cpu().numpy().view(np.uint32))
            self.args = og.default_arguments(fnameb=path, sort=sort, pushpull=2)
            self.lib.initializeMersenneState(ctypes.byref(self.args.mt19937var), 27491095)
            self.graph = self.lib.graphCSRPreProcessingStep(ctypes.byref(self.args))
        finally:
            os.unlink(path)

    def __del__(self):
        if getattr(self, "graph", None):
            self.lib.graphCSRFree(self.graph)
            self.graph = None


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "batch":
        nv, off, src, dst, roots = _batch_edges(case, seed)
        st["batch"] = og.GraphBatch(og.load(False), nv, off, src.cpu().numpy().view(np.uint32),
                                    dst.cpu().numpy().view(np.uint32))
        st["roots"] = roots
        V = int(st["batch"].offsets[-1])
        st["parents"] = torch.empty(V, dtype=torch.int32, device="cuda")
        st["distances"] = torch.empty(V, dtype=torch.int32, device="cuda")
        st["ranks"] = torch.empty(V, dtype=torch.float32, device="cuda")
        st["keep"] = _Closer(st["batch"])
        return st
    V, src, dst, w, gen = _edges(case, seed)
    if kind == "dropin":
        src[0] = V - 1  # an edge file's vertex count is its largest id + 1
        st["root"] = _roots(src, V, 1, gen)[0]
        st["host"] = _HostGraph(src, dst, case["sort"])
        st["host"].args.source = st["root"]
        return st
    st["graph"] = og.load(w is not None).device_graph()
    st["V"] = V
    if kind in ("flow", "build"):
        st.update(src=src, dst=dst, w=w)
    else:
        st["graph"].build(src, dst, V, case.get("sort", 0), weight=w)
    if kind in ("flow", "bfs"):
        st["root"] = _roots(src, V, 1, gen)[0]
        st["parents"] = torch.empty(V, dtype=torch.int32, device="cuda")
        st["distances"] = torch.empty(V, dtype=torch.int32, device="cuda")
    if kind in ("flow", "pagerank"):
        st["ranks"] = torch.empty(V, dtype=torch.float32, device="cuda")
    if kind == "spmv":
        st["x"] = torch.empty(V, dtype=torch.float32, device="cuda")
        st["y"] = torch.empty(V, dtype=torch.float32, device="cuda")
    if kind == "msbfs":
        st["roots"] = _roots(src, V, case["roots"], gen)
        st["depths"] = torch.empty(V * 64, dtype=torch.int16, device="cuda")
    if kind == "ppr":
        st["seeds"] = _roots(src, V, case["seeds"], gen)
        st["ranks"] = torch.empty(V * 32, dtype=torch.float32, device="cuda")
    return st


class _Closer:
    """Closes a GraphBatch when its state goes."""

    def __init__(self, batch):
        self.batch = batch

    def __del__(self):
        self.batch.close()


# --------------------------------------------------------------------- run --

def _bfs(st):
    info = st["graph"].bfs(st["root"], st["parents"], st["distances"], mode=2)
    return {"distances": st["distances"], **{k: info[k] for k in ("iteration", "processed_nodes", "td_steps", "bu_steps",
                                                                  "reached", "reached_out_edges", "edges_examined")}}


def _csr(st):
    out = {}
    for name, inverse in (("forward", False), ("inverse", True)):
        v = st["graph"].view(inverse)
        out[name] = {"src": v.src, "dst": v.dst, "weight": v.weight, "out_degree": v.out_degree,
                     "in_degree": v.in_degree, "edges_idx": v.edges_idx}
        for t in out[name].values():
            if t is not None:
                t.graph = st["graph"]  # the arrays are the graph's own: whoever holds one holds the graph
    return out


def _dropin(st):
    host = st["host"]
    lib = host.lib
    stats = lib.breadthFirstSearchGraphCSR(ctypes.byref(host.args), host.graph)
    s = stats.contents
    out = {"distances": og.as_numpy(s.distances, s.num_vertices, np.uint32).view(np.int32),
           "processed_nodes": int(s.processed_nodes), "iteration": int(s.iteration)}
    lib.freeBFSStats(stats)
    return out


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "flow":
        st["graph"].build(st["src"], st["dst"], st["V"], case["sort"], weight=st["w"])
        found = _bfs(st)
        info = st["graph"].pagerank(st["ranks"], mode=0, max_iterations=case["iters"], epsilon=1e-4)
        return {"csr": _csr(st), "bfs": found, "ranks": st["ranks"], "iterations": info["iterations"]}
    if kind == "build":
        st["graph"].build(st["src"], st["dst"], st["V"], case["sort"], weight=st["w"])
        return _csr(st)
    if kind == "bfs":
        return _bfs(st)
    if kind == "dropin":
        return _dropin(st)
    if kind == "pagerank":
        info = st["graph"].pagerank(st["ranks"], mode=case["mode"], max_iterations=case["iters"], epsilon=1e-4)
        return {"ranks": st["ranks"], "iterations": info["iterations"], "error": info["error_total"]}
    if kind == "spmv":
        st["graph"].spmv(st["x"], st["y"], mode=case["mode"], iterations=case["iters"])
        return {"x": st["x"], "y": st["y"]}
    if kind == "msbfs":
        info = st["graph"].msbfs(st["roots"], st["depths"])
        return {"depths": st["depths"], "levels": info["levels"], "reached_pairs": info["reached_pairs"]}
    if kind == "ppr":
        info = st["graph"].ppr(st["seeds"], st["ranks"], max_iterations=case["iters"])
        return {"ranks": st["ranks"], "executed": info["executed"]}
    found = st["batch"].bfs(st["roots"], st["parents"], st["distances"])
    _, per = st["batch"].pagerank(st["ranks"], max_iterations=case["iters"], epsilon=1e-4)
    return {"distances": st["distances"], "reached": found["reached"], "ranks": st["ranks"],
            "iterations": np.array([p["iterations"] for p in per], dtype=np.int64)}


# -------------------------------------------------------------------- work --

def work(case):
    kind = case["kind"]
    if kind == "batch":
        mean_v = sum(1 << s for s in range(case["lo"], case["hi"] + 1)) / (case["hi"] - case["lo"] + 1)
        V = case["graphs"] * mean_v
        E = V * (case["ef_lo"] + case["ef_hi"]) / 2
        return {"bytes": 24 * V + case["iters"] * (4 * E + 24 * V), "flops": case["iters"] * E}
    V = _vertices(case)
    E = case["E"] if case["graph"] != "grid" else 4 * V
    edge = 12 if case.get("weighted") else 8
    # the edge list in, both directions' edges and vertex arrays out
    build = 3 * edge * E + 24 * V
    # a row and at least one neighbour id per vertex, out-degrees in; parents
    # and depths out (a grid's search reads every edge)
    bfs = 24 * V + (4 * E if case["graph"] == "grid" else 0)
    # ids once per iteration; contribs, degrees and rows in, ranks and contribs out
    iters = case.get("iters", 1)
    pull = iters * (4 * E + 24 * V)
    if kind == "flow":
        return {"bytes": build + bfs + pull, "flops": iters * E}
    if kind == "build":
        return {"bytes": build, "flops": 0}
    if kind in ("bfs", "dropin"):
        return {"bytes": bfs, "flops": 0}
    if kind == "pagerank":
        return {"bytes": pull, "flops": iters * E}
    if kind == "spmv":
        return {"bytes": iters * ((edge - 4) * E + 16 * V), "flops": 2 * iters * E}
    if kind == "msbfs":
        return {"bytes": 4 * E + (24 + 2 * 64) * V, "flops": 0}
    # 32 ranks of a vertex in and out, its contribs in once
    return {"bytes": iters * (4 * E + 3 * 128 * V), "flops": iters * 32 * E}


# ------------------------------------------------------------------- exact --

def _pull64(src, dst, size, first, iters, eps):
    """Ranks after the iterations of the rule "stop when nothing changes by
    eps", per part of a union (size: vertices of each vertex's part, first:
    the parts' offsets), in 64 bits."""
    V = size.numel()
    deg = torch.zeros(V, dtype=torch.float64, device="cuda").index_add_(
        0, src.long(), torch.ones(src.numel(), dtype=torch.float64, device="cuda"))
    pr = torch.full((V,), BASE, dtype=torch.float64, device="cuda")
    part = torch.repeat_interleave(torch.arange(len(first) - 1, device="cuda"),
                                   torch.tensor([b - a for a, b in zip(first, first[1:])], device="cuda"))
    on = torch.ones(len(first) - 1, dtype=torch.bool, device="cuda")
    s, d = src.long(), dst.long()
    err = 0.0
    for _ in range(iters):
        c = torch.where(deg > 0, pr / deg.clamp(min=1), torch.zeros_like(pr))
        new = BASE + DAMP * torch.zeros_like(pr).index_add_(0, d, c[s])
        new = torch.where(on[part], new, pr)
        change = (new - pr).abs()
        pr = new
        err = float((change / size).sum())
        worst = torch.zeros(len(first) - 1, dtype=torch.float64, device="cuda").scatter_reduce_(0, part, change, "amax")
        on &= worst >= eps
        if not bool(on.any()):
            break
    return pr / size, err


def exact(case, seed):
    kind = case["kind"]
    if kind in ("bfs", "dropin", "msbfs", "build"):
        return None
    if kind == "batch":
        nv, off, src, dst, _ = _batch_edges(case, seed)
        first = [0] + np.cumsum(nv).tolist()
        shift = torch.repeat_interleave(torch.tensor(first[:-1], device="cuda"),
                                        torch.tensor([b - a for a, b in zip(off, off[1:])], device="cuda"))
        size = torch.repeat_interleave(torch.tensor(nv, device="cuda"), torch.tensor(nv, device="cuda")).double()
        ranks, _ = _pull64(src.long() + shift, dst.long() + shift, size, first, case["iters"], 1e-4)
        return {"distances": None, "reached": None, "ranks": ranks, "iterations": None}
    V, src, dst, w, gen = _edges(case, seed)
    size = torch.full((V,), float(V), dtype=torch.float64, device="cuda")
    if kind in ("flow", "pagerank"):
        ranks, err = _pull64(src, dst, size, [0, V], case["iters"], 1e-4)
        if kind == "flow":
            return {"csr": None, "bfs": None, "ranks": ranks, "iterations": None}
        return {"ranks": ranks, "iterations": None, "error": err}
    deg = torch.zeros(V, dtype=torch.float64, device="cuda").index_add_(
        0, src.long(), torch.ones(src.numel(), dtype=torch.float64, device="cuda"))
    if kind == "spmv":
        x = torch.where(deg > 0, 1.0 / deg.clamp(min=1), torch.full_like(deg, float(np.float32(0.001))))
        wt = w.double() if w is not None else float(np.float32(0.0001))
        y = torch.zeros_like(x).index_add_(0, dst.long(), x[src.long()] * wt)
        return {"x": x, "y": y * case["iters"]}
    seeds = _roots(src, V, case["seeds"], gen)
    s, d = src.long(), dst.long()
    out = torch.zeros(V, 32, dtype=torch.float64, device="cuda")
    for k, v in enumerate(seeds):
        pr = torch.zeros(V, dtype=torch.float64, device="cuda")
        pr[v] = 1.0
        for _ in range(case["iters"]):
            c = torch.where(deg > 0, pr / deg.clamp(min=1), torch.zeros_like(pr))
            pr = DAMP * torch.zeros_like(pr).index_add_(0, d, c[s])
            pr[v] += BASE
        out[:, k] = pr
    return {"ranks": out.view(-1), "executed": None}
