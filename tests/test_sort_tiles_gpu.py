"""The radix pass at the edges of its tiles (4096 keys) and warps, for digits of
seven and eight bits, with and without weights: the sorted list equals numpy's
stable sort, and a build's rows equal the oracle's."""
import numpy as np
import pytest

from test_build_gpu import dev, host

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 33, 511, 513, 4095, 4096, 4097, 8192, 12289, 40961]


def edges(n, V, seed, skew):
    rng = np.random.default_rng(seed)
    s = rng.integers(0, V, n).astype(np.uint32)
    d = rng.integers(0, V, n).astype(np.uint32)
    if skew:  # most keys share a digit
        s[rng.random(n) < 0.9] = V - 1
    return s, d, rng.uniform(1, 256, n).astype(np.float32)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", SIZES)
def test_sort_edges_tiles(torch_cuda, lib, n, weighted):
    for V, skew in ((1 << 30, False), (300, True), (1, False)):
        s, d, w = edges(n, V, n, skew)
        ts, td, tw = dev(torch_cuda, s), dev(torch_cuda, d), torch_cuda.from_numpy(w).cuda()
        for sort_type in (0, 1):
            os_, od, ow = torch_cuda.empty_like(ts), torch_cuda.empty_like(td), torch_cuda.empty_like(tw)
            torch_cuda.cuda.synchronize()
            lib.check(lib.ogb_sort_edges(ts.data_ptr(), td.data_ptr(), tw.data_ptr() if weighted else None, n, sort_type,
                                         os_.data_ptr(), od.data_ptr(), ow.data_ptr() if weighted else None, None))
            order = np.lexsort((d, s)) if sort_type else np.argsort(s, kind="stable")
            assert np.array_equal(host(os_).view(np.uint32), s[order])
            assert np.array_equal(host(od).view(np.uint32), d[order])
            if weighted:
                assert np.array_equal(host(ow, np.float32), w[order])


@pytest.mark.parametrize("V", [2, 127, 128, 129, 256, 257, 16384, 16385, 1 << 21])
def test_build_digit_widths(torch_cuda, lib, oracle, V):
    s, d, w = edges(9001, V, V, True)
    exp = oracle.build(s, d, V, 0, w)
    g = lib.device_graph()
    g.build(dev(torch_cuda, s), dev(torch_cuda, d), V, 0, weight=torch_cuda.from_numpy(w).cuda())
    for tag, inv in (("f", False), ("i", True)):
        v = g.view(inv)
        for name, arr in (("src", v.src), ("dst", v.dst), ("outdeg", v.out_degree), ("idx", v.edges_idx)):
            assert np.array_equal(host(arr).view(np.uint32), exp[f"{tag}_{name}"]), (tag, name)
        assert np.array_equal(host(v.weight, np.float32), exp[f"{tag}_w"]), tag
    g.close()
