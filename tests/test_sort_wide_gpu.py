"""The sorts of 2^30 edges and more use 8-byte look-back words: here at sizes
around the tiles of a pass, with and without weights, by one key and by two, built
graphs against the oracle's."""
import numpy as np
import pytest

from test_build_gpu import dev, host
from test_sort_tiles_gpu import edges

pytestmark = pytest.mark.gpu

WIDE_LOOKBACK = 3


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("sort_type", [0, 1])
@pytest.mark.parametrize("n,V", [(1, 1), (4095, 300), (4097, 70_000), (40_961, 128), (600_001, 1 << 18)])
def test_build(torch_cuda, lib, oracle, n, V, sort_type, weighted):
    s, d, w = edges(n, V, n, True)
    exp = oracle.build(s, d, V, sort_type, w if weighted else None)
    g = lib.device_graph()
    lib.check(lib.ogb_graph_test_option(g.handle, WIDE_LOOKBACK, 1))
    g.build(dev(torch_cuda, s), dev(torch_cuda, d), V, sort_type,
            weight=torch_cuda.from_numpy(w).cuda() if weighted else None)
    for tag, inv in (("f", False), ("i", True)):
        v = g.view(inv)
        for name, arr in (("src", v.src), ("dst", v.dst), ("outdeg", v.out_degree), ("idx", v.edges_idx)):
            assert np.array_equal(host(arr).view(np.uint32), exp[f"{tag}_{name}"]), (tag, name)
        if weighted:
            assert np.array_equal(host(v.weight, np.float32), exp[f"{tag}_w"]), tag
    g.close()
