"""A sort whose look-back gave up: a build reports it, whichever of its sorts it
was, and PageRank's renumbering, which decides only where values are kept, falls
back to the ids as they are."""
import numpy as np
import pytest

from test_build_gpu import dev, host
from test_pagerank_gpu import bins

pytestmark = pytest.mark.gpu

SORT_GIVES_UP = 1


def test_pagerank_without_the_renumbering(torch_cuda, lib, oracle, graphs):
    s, d, _, V = graphs("rmat", scale=13, ef=16, seed=5)
    g = oracle.build(s, d, V, 0)
    dg = lib.device_graph()
    dg.build(dev(torch_cuda, s), dev(torch_cuda, d), V, 0)
    lib.check(lib.ogb_graph_test_option(dg.handle, SORT_GIVES_UP, 1))
    oracle.set_gpu_order(*bins(lib))
    ranks = torch_cuda.empty(V, dtype=torch_cuda.float32, device="cuda")
    for _ in range(2):
        dg.pagerank(ranks, mode=0, max_iterations=6, epsilon=0.0)
        er, _ = oracle.pagerank(g, 2, 6, 0.0)
        assert np.array_equal(host(ranks, np.float32).view(np.uint32), er.view(np.uint32))
    dg.close()


@pytest.mark.parametrize("sort_type", [0, 1])
def test_build_reports(torch_cuda, lib, og, oracle, graphs, sort_type):
    s, d, _, V = graphs("rmat", scale=12, ef=16, seed=1)
    ts, td = dev(torch_cuda, s), dev(torch_cuda, d)
    dg = lib.device_graph()
    for first in (1, 2):  # the first sort, both
        lib.check(lib.ogb_graph_test_option(dg.handle, SORT_GIVES_UP, first))
        with pytest.raises(og.OgbError, match="look-back"):
            dg.build(ts, td, V, sort_type)
        dg.build(ts, td, V, sort_type)
        exp = oracle.build(s, d, V, sort_type)
        for tag, inv in (("f", False), ("i", True)):
            v = dg.view(inv)
            assert np.array_equal(host(v.src).view(np.uint32), exp[f"{tag}_src"])
            assert np.array_equal(host(v.dst).view(np.uint32), exp[f"{tag}_dst"])
    dg.close()
