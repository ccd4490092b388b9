"""Rows around the lengths at which their sums are cut: personalized PageRank's
chunks (512 in-edges), the row classes of SPMV and data-driven pull (32, 2048 and
chunks of 8192), and a graph whose medium rows make more units of PageRank pull
than the kernel has warps, so that the rest are handed out by a counter."""
import numpy as np
import pytest

from test_build_gpu import dev, host
from test_pagerank_gpu import bins

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 32, 33, 511, 512, 513, 1024, 1025, 2047, 2048, 2049, 8191, 8192, 8193, 16384, 16385]


def graph(torch, lib, oracle, weighted):
    V = 3000
    rng = np.random.default_rng(4)
    d = np.concatenate([np.full(n, 7 * i) for i, n in enumerate(LENGTHS)] + [rng.integers(200, V, 4000)])
    s = rng.integers(0, V, len(d))
    order = rng.permutation(len(d))
    s, d = s[order].astype(np.uint32), d[order].astype(np.uint32)
    w = rng.uniform(1, 256, len(s)).astype(np.float32) if weighted else None
    g = oracle.build(s, d, V, 0, w)
    dg = lib.device_graph()
    dg.build(dev(torch, s), dev(torch, d), V, 0, weight=dev(torch, w))
    return g, dg, V


@pytest.mark.parametrize("weighted", [False, True])
def test_spmv_and_data_driven_pull(torch_cuda, lib, libw, oracle, weighted):
    torch = torch_cuda
    g, dg, V = graph(torch, libw if weighted else lib, oracle, weighted)
    oracle.set_gpu_order()
    x = torch.empty(V, dtype=torch.float32, device="cuda")
    y = torch.empty(V, dtype=torch.float32, device="cuda")
    for iters in (1, 3):
        dg.spmv(x, y, mode=0, iterations=iters)
        _, ey = oracle.spmv(g, 0, iters, weighted=weighted, gpu_order=True)
        assert np.array_equal(host(y, np.float32).view(np.uint32), ey.view(np.uint32)), iters
    dg.pagerank(x, mode=6, max_iterations=12, epsilon=1e-4)
    er, _ = oracle.pagerank_dd(g, 6, 12, 1e-4, gpu_order=True)
    assert np.array_equal(host(x, np.float32).view(np.uint32), er.view(np.uint32))
    dg.close()


@pytest.mark.parametrize("nseeds", [1, 5, 32])
def test_personalized(torch_cuda, lib, oracle, nseeds):
    """Against the iteration in 64 bits: each rank is a sum of positive terms, so an
    iteration adds at most (n + 4) 2^-24 of relative error, n its in-edges."""
    torch = torch_cuda
    g, dg, V = graph(torch, lib, oracle, False)
    seeds = np.random.default_rng(nseeds).permutation(V)[:nseeds].astype(np.uint32)
    ranks = torch.empty(V * 32, dtype=torch.float32, device="cuda")
    iters = 4
    dg.ppr(seeds, ranks, max_iterations=iters)
    got = host(ranks, np.float32).reshape(V, 32).astype(np.float64)
    deg = g["f_outdeg"].astype(np.float64)
    damp, base = float(np.float32(0.85)), float(np.float32(1.0) - np.float32(0.85))
    bound = iters * (float(g["i_outdeg"].max()) + 4) * 2.0 ** -24
    for k, v in enumerate(seeds):
        pr = np.zeros(V)
        pr[v] = 1.0
        for _ in range(iters):
            c = np.divide(pr, deg, out=np.zeros(V), where=deg > 0)
            pr = damp * np.bincount(g["f_dst"], weights=c[g["f_src"]], minlength=V)
            pr[v] += base
        assert np.all(np.abs(got[:, k] - pr) <= bound * pr + 1e-30), k
    assert np.all(got[:, nseeds:] == 0.0)
    dg.close()


def test_pull_units_beyond_the_warps(torch_cuda, lib, oracle):
    torch = torch_cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    V = 40_000
    E = 80 * sms * 32 * 8  # units of 256 edges for 2.5 times the kernel's warps, rows of about 75 edges
    rng = np.random.default_rng(8)
    s, d = rng.integers(0, V, (2, E)).astype(np.uint32)
    g = oracle.build(s, d, V, 0)
    dg = lib.device_graph()
    dg.build(dev(torch, s), dev(torch, d), V, 0)
    oracle.set_gpu_order(*bins(lib))
    ranks = torch.empty(V, dtype=torch.float32, device="cuda")
    for iters in (1, 3):
        dg.pagerank(ranks, mode=0, max_iterations=iters, epsilon=0.0)
        er, _ = oracle.pagerank(g, 2, iters, 0.0)
        assert np.array_equal(host(ranks, np.float32).view(np.uint32), er.view(np.uint32)), iters
    dg.close()
