"""SPMV and the data-driven PageRank modes on device copies of host GraphCSRs:
one made while a .csr file is read, one made at the first call on a GraphCSR that
the library has not seen.  Such a copy has no array of edge sources, so the self
loops that data-driven push counts come from the out-rows; the crafted graph has
rows around the lengths at which their count goes from a lane to a chunk, and its
active counts are known (`crossings`)."""
import ctypes as C

import numpy as np
import pytest

from test_build_gpu import host
from test_dd_gpu import DD_SEQ_TOL, push_bound

pytestmark = pytest.mark.gpu

# (self loops, other out-edges) of a vertex
ROWS = [(1, 0), (0, 3), (2, 1), (0, 0), (31, 1), (16, 17), (32, 0), (33, 0), (20, 13), (500, 523), (512, 512), (513, 512),
        (1023, 0), (1024, 0), (1025, 0), (1, 1024), (2047, 2), (3000, 2000), (5, 5)] * 5


def loops_graph():
    ss, dd, at = [], [], len(ROWS)
    for v, (k, m) in enumerate(ROWS):
        ss.append(np.full(k + m, v))
        dd.append(np.concatenate([np.full(k, v), np.arange(at, at + m)]))
        at += m
    s, d = np.concatenate(ss), np.concatenate(dd)
    d[-1] = at  # the vertex count is the largest id + 1
    order = np.random.default_rng(1).permutation(len(s))
    return s[order].astype(np.uint32), d[order].astype(np.uint32), None


copies = []  # kept: the library knows a GraphCSR by its address


class Uploaded:
    """The device copy of a GraphCSR read from a .csr file ("file"), or of one at
    an address that has no copy yet ("call")."""

    def __init__(self, og, lib, tmp_path, edges, weighted, how):
        s, d, w = edges
        path = str(tmp_path / ("g.wbin" if weighted else "g.bin"))
        og.write_edge_file(path, s, d, w if weighted else None)
        a = og.default_arguments(fnameb=path, sort=0, weighted=1 if weighted else 0)
        lib.initializeMersenneState(C.byref(a.mt19937var), 27491095)
        built = lib.graphCSRPreProcessingStep(C.byref(a))
        lib.writeToBinFileGraphCSR(str(tmp_path / "g").encode(), built)
        lib.graphCSRFree(built)
        self.lib, self.graph = lib, lib.readFromBinFileGraphCSR(str(tmp_path / "g.csr").encode())
        self.arrays = og.graph_arrays(self.graph)
        self.V = self.arrays["num_vertices"]
        at = self.graph
        if how == "call":
            copies.append(type(self.graph.contents)())
            C.memmove(C.byref(copies[-1]), self.graph, C.sizeof(copies[-1]))
            at = C.pointer(copies[-1])
        self.dg = og.DeviceGraph(lib, lib.ogb_graph_of(C.cast(at, C.c_void_p)), owned=False)
        assert self.dg.handle

    def close(self):
        self.dg.close()
        self.lib.graphCSRFree(self.graph)


def crossings(eps):
    """Bounds of the first iteration's active count.  A vertex with k self loops
    among its k + m out-edges has residual r = c k / (k + m), c = 0.15 * 0.85, and
    each self loop adds delta = 0.85 r / (k + m): one crossing if r <= eps <= r + k
    delta.  A vertex that one of them pushes to has c / (k + m), or nothing if it
    took its own residual before the push: both orders are allowed."""
    lo = hi = 0
    for k, m in ROWS:
        n = max(k + m, 1)
        r = 0.1275 * k / n
        delta = 0.85 * r / n
        assert min(abs(r - eps), abs(r + k * delta - eps)) > 1e-6
        lo, hi = lo + (r <= eps <= r + k * delta), hi + (r <= eps <= r + k * delta)
        before, after = 0.1275 / n <= eps <= 0.1275 / n + delta, delta >= eps
        lo, hi = lo + m * (before and after), hi + m * (before or after)
    return lo, hi


@pytest.mark.parametrize("how", ["file", "call"])
def test_self_loops_counted(torch_cuda, og, lib, oracle, tmp_path, how):
    u = Uploaded(og, lib, tmp_path, loops_graph(), False, how)
    ranks = torch_cuda.empty(u.V, dtype=torch_cuda.float32, device="cuda")
    crossed = set()
    for eps in (0.01, 0.05, 0.08, 0.1, 0.13, 0.18, 0.22):
        u.dg.pagerank(ranks, mode=7, max_iterations=4, epsilon=eps)
        _, act = u.dg.pagerank_history()
        lo, hi = crossings(eps)
        assert lo <= act[0] <= hi and not np.any(act[1:]), eps
        _, info = oracle.pagerank_dd(u.arrays, 7, 4, eps)
        assert lo <= info["active_hist"][0] <= hi
        crossed.add(int(act[0]))
    assert len(crossed) > 3  # the counts tell the thresholds apart
    u.close()


@pytest.mark.parametrize("how", ["file", "call"])
@pytest.mark.parametrize("weighted", [False, True])
def test_spmv_and_data_driven(torch_cuda, og, lib, libw, oracle, tmp_path, weighted, how):
    torch = torch_cuda
    u = Uploaded(og, libw if weighted else lib, tmp_path, og.generate_rmat(12, 16, 6, weighted=True), weighted, how)
    g, V = u.arrays, u.V
    oracle.set_gpu_order()
    x = torch.empty(V, dtype=torch.float32, device="cuda")
    y = torch.empty(V, dtype=torch.float32, device="cuda")
    u.dg.spmv(x, y, mode=0, iterations=5)
    ex, ey = oracle.spmv(g, 0, 5, weighted=weighted, gpu_order=True)
    assert np.array_equal(host(x, np.float32).view(np.uint32), ex.view(np.uint32))
    assert np.array_equal(host(y, np.float32).view(np.uint32), ey.view(np.uint32))
    u.dg.spmv(x, y, mode=1, iterations=5)
    _, sy = oracle.spmv(g, 1, 5, weighted=weighted)
    rel = np.abs(host(y, np.float32).astype(np.float64) - sy) / np.maximum(np.abs(sy), 1e-30)
    assert np.all(rel <= push_bound(g, 5)), float(rel.max())
    u.dg.pagerank(x, mode=6, max_iterations=30, epsilon=1e-4)
    er, _ = oracle.pagerank_dd(g, 6, 30, 1e-4, gpu_order=True)
    assert np.array_equal(host(x, np.float32).view(np.uint32), er.view(np.uint32))
    for mode in (7, 8):
        u.dg.pagerank(x, mode=mode, max_iterations=100, epsilon=1e-6)
        seq, _ = oracle.pagerank_dd(g, mode, 100, 1e-6)
        assert float(np.abs(host(x, np.float32).astype(np.float64) - seq).sum()) <= DD_SEQ_TOL, mode
    u.close()
