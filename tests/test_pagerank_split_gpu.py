"""PageRank pull at the edges of its work split: row lengths around the class
bounds (32, 2048), the copy's piece bounds (1024, 4096) and the chunk bound
(8192), vertex counts around the warp, tile and wide-light bounds, bit-exact
against the oracle in the kernel's summation order; and a batch of graphs whose
sizes lie around the piece bound of the per-graph reduction."""
import numpy as np
import pytest

from test_build_gpu import dev, host
from test_pagerank_gpu import bins

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4097, 8191, 8192, 8193, 16385]


def edges(V, seed):
    """A row of each length (as far as V goes) and a few edges everywhere."""
    rng = np.random.default_rng(seed)
    dst = [np.full(n, (i * 7919) % V, np.uint32) for i, n in enumerate(LENGTHS)]
    dst.append(rng.integers(0, V, 3 * min(V, 50_000)).astype(np.uint32))
    dst = np.concatenate(dst)
    src = rng.integers(0, V, len(dst)).astype(np.uint32)
    order = rng.permutation(len(dst))
    return src[order], dst[order]


@pytest.mark.parametrize("V", [1, 31, 33, 2047, 2049, 4097, 606_207, 606_209])
def test_pull_bitexact_at_split_edges(torch_cuda, lib, oracle, V):
    s, d = edges(V, V)
    g = oracle.build(s, d, V, 0)
    dg = lib.device_graph()
    dg.build(dev(torch_cuda, s), dev(torch_cuda, d), V, 0)
    oracle.set_gpu_order(*bins(lib))
    ranks = torch_cuda.empty(V, dtype=torch_cuda.float32, device="cuda")
    for iters in (1, 6):
        dg.pagerank(ranks, mode=0, max_iterations=iters, epsilon=0.0)
        er, _ = oracle.pagerank(g, 2, iters, 0.0)
        assert np.array_equal(host(ranks, np.float32).view(np.uint32), er.view(np.uint32)), iters
    dg.close()


def test_batch_piece_edges(torch_cuda, lib, oracle, og):
    nv = [1, 0, 2047, 2048, 2049, 4097]
    parts = [edges(v, v) if v else (np.zeros(0, np.uint32),) * 2 for v in nv]
    off = np.concatenate([[0], np.cumsum([len(p[0]) for p in parts])])
    b = og.GraphBatch(lib, nv, off, np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts]))
    oracle.set_gpu_order(*bins(lib))
    ranks = torch_cuda.empty(sum(nv), dtype=torch_cuda.float32, device="cuda")
    for iters, eps in ((8, 0.0), (60, 1e-4)):
        _, per = b.pagerank(ranks, max_iterations=iters, epsilon=eps)
        got = host(ranks, np.float32)
        for i, v in enumerate(nv):
            if v == 0:
                assert per[i]["executed"] == 1 and per[i]["converged"] == 1
                continue
            er, ei = oracle.pagerank(oracle.build(*parts[i], v, 0), 2, iters, eps)
            lo = int(b.offsets[i])
            assert np.array_equal(got[lo:lo + v].view(np.uint32), er.view(np.uint32)), (i, iters)
            assert per[i]["iterations"] == ei["iterations"], (i, iters)
    b.close()
