"""Runs of narrow top-down steps (small lists of low out-degree, taken by one
cluster of CTAs) against the oracle: layer widths and out-degrees around the
bounds at which a search enters and leaves such a run, lists that grow past
them and shrink again, layers without out-edges, and searches from several
roots at once."""
import numpy as np
import pytest

from test_bfs_gpu import check_parents
from test_build_gpu import dev, host

pytestmark = pytest.mark.gpu


def layered(widths, degree, seed):
    """Layers of the given widths; every vertex has `degree` out-edges into the
    next layer, every vertex of which has at least one in-edge if they suffice."""
    rng = np.random.default_rng(seed)
    first = np.concatenate([[0], np.cumsum(widths)])
    ss, dd = [], []
    for i in range(len(widths) - 1):
        s = np.repeat(np.arange(first[i], first[i + 1]), degree)
        d = first[i + 1] + (np.arange(len(s)) + rng.integers(0, widths[i + 1])) % widths[i + 1]
        ss.append(s)
        dd.append(d)
    s, d = np.concatenate(ss), np.concatenate(dd)
    perm = rng.permutation(first[-1])  # vertex ids in no order
    order = rng.permutation(len(s))
    return perm[s][order].astype(np.uint32), perm[d][order].astype(np.uint32), int(first[-1]), int(perm[0])


SHAPES = {
    "w700-d4": ([1, 4, 16, 64] + [700] * 30, 4),
    "enter-2047": ([1, 8, 64, 512] + [2047] * 12, 8),
    "enter-2048": ([1, 8, 64, 512] + [2048] * 12, 8),
    "enter-2049": ([1, 8, 64, 512] + [2049] * 12, 8),
    "d32": ([1] + [32] * 12 + [1000] * 6, 32),
    "d33": ([1] + [33] * 12 + [1000] * 6, 33),
    "queue-2048x32": ([1] + [30] * 8 + [900, 2048, 2048, 2048, 20000, 30, 30, 30, 30, 30, 30], 32),
    "cap-8192": ([1] + [5] * 8 + [15, 45, 135, 405, 1215, 3645, 8192, 8192, 8193, 9000, 20, 20, 20, 20, 20, 20], 3),
    "grow-shrink": ([1] + [2] * 8 + [4, 8, 16, 32, 64, 128, 256, 512, 1024, 2048, 4096, 8192, 16384, 30000] +
                    [64] * 10 + [300] * 10, 2),
    "one": ([1] * 60, 1),
}


def check(torch, lib, oracle, s, d, V, root, modes=(2, 1)):
    g = oracle.build(s, d, V, 0)
    dg = lib.device_graph()
    dg.build(dev(torch, s), dev(torch, d), V, 0)
    par_t = torch.empty(V, dtype=torch.int32, device="cuda")
    dist_t = torch.empty(V, dtype=torch.int32, device="cuda")
    for mode in modes:
        info = dg.bfs(root, par_t, dist_t, mode=mode)
        _, edist, est = oracle.bfs(g, root, mode)
        par, dist = host(par_t, np.int32), host(dist_t)
        assert np.array_equal(dist, edist), mode
        for k in ("iteration", "processed_nodes", "td_steps", "bu_steps", "reached", "reached_out_edges"):
            assert info[k] == est[k], (mode, k)
        trace = dg.bfs_trace()
        assert [t["direction"] for t in trace] == list(est["dirs"][:len(trace)])
        assert sum(t["discovered"] for t in trace) + 1 == est["processed_nodes"]
        assert len(dg.bfs_features()) == len(trace)
        check_parents(g, root, par, dist)
    dg.close()


@pytest.mark.parametrize("shape", list(SHAPES))
def test_layers(torch_cuda, lib, oracle, shape):
    widths, degree = SHAPES[shape]
    s, d, V, root = layered(widths, degree, 3)
    check(torch_cuda, lib, oracle, s, d, V, root)
    # the same beside many edges the root does not reach: the switch stays top-down for longer
    rng = np.random.default_rng(5)
    more = rng.integers(0, 20_000, (2, 400_000)) + V
    check(torch_cuda, lib, oracle, np.concatenate([s, more[0].astype(np.uint32)]),
          np.concatenate([d, more[1].astype(np.uint32)]), V + 20_000, root)


def test_grid_and_batch(torch_cuda, lib, oracle, og, graphs):
    torch = torch_cuda
    s, d, _, V = graphs("grid", side=150, p=0.001, seed=2)
    check(torch, lib, oracle, s, d, V, V // 3)
    parts = [(s, d, V)] + [layered([1] + [w] * 20, 3, w)[:3] for w in (1, 7, 300)]
    nv = [p[2] for p in parts]
    off = np.concatenate([[0], np.cumsum([len(p[0]) for p in parts])])
    b = og.GraphBatch(lib, nv, off, np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts]))
    roots = [V - 1, 0, 1, 2]
    par = torch.empty(sum(nv), dtype=torch.int32, device="cuda")
    dist = torch.empty(sum(nv), dtype=torch.int32, device="cuda")
    info = b.bfs(roots, par, dist)
    reached = 0
    for i, (ps, pd, v) in enumerate(parts):
        epar, edist, _ = oracle.bfs(oracle.build(ps, pd, v, 0), roots[i], 2)
        lo = int(b.offsets[i])
        assert np.array_equal(host(dist)[lo:lo + v], edist), i
        reached += int((epar >= 0).sum())
    assert info["reached"] == reached
    b.close()
