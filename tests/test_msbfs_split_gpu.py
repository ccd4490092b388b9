"""Multi-source BFS at the edges of its work split: out-rows around the piece
bound of a push level (512), frontiers around a warp's 32 vertices, vertex counts
around the tiles of the dense pass, and searches of one level more and less than
the levels launched between two looks of the host."""
import numpy as np
import pytest

from test_batch_gpu import check_lanes
from test_build_gpu import dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extra", [0, 1, 200])
@pytest.mark.parametrize("lengths", [[0, 1, 511, 512, 513, 1023, 1024, 1025, 1537], [3] * 31, [3] * 32, [600] * 33])
def test_push_rows(torch_cuda, lib, oracle, lengths, extra):
    rng = np.random.default_rng(len(lengths) + extra)
    n = len(lengths)
    V = 4096 + extra
    # root -> the hubs, each hub -> its targets; a chain beside it keeps E large
    s = np.concatenate([np.zeros(n, np.int64)] + [np.full(k, 1 + i) for i, k in enumerate(lengths)] +
                       [rng.integers(2000, V, 60_000)])
    d = np.concatenate([np.arange(1, n + 1)] + [rng.integers(100, V, k) for k in lengths] +
                       [rng.integers(2000, V, 60_000)])
    s, d = s.astype(np.uint32), d.astype(np.uint32)
    run(torch_cuda, lib, oracle, s, d, V, [0, 1, min(3, n), V - 1, 0])


@pytest.mark.parametrize("levels", [1, 2, 3, 4, 5, 7, 8, 9])
def test_level_counts(torch_cuda, lib, oracle, levels):
    s = np.arange(levels, dtype=np.uint32)
    run(torch_cuda, lib, oracle, s, s + 1, levels + 1, [0, levels])


def run(torch, lib, oracle, s, d, V, roots):
    g = oracle.build(s, d, V, 0)
    dg = lib.device_graph()
    dg.build(dev(torch, s), dev(torch, d), V, 0)
    depth_t = torch.empty(V * 64, dtype=torch.int16, device="cuda")
    info = dg.msbfs(roots, depth_t)
    depths = host(depth_t, np.int16).view(np.uint16).reshape(V, 64)
    check_lanes(oracle, g, roots, depths)
    assert info["reached_pairs"] == int((depths[:, :len(roots)] != 0xFFFF).sum())
    # the last level finds nothing, and is counted
    assert info["levels"] == int(depths[:, :len(roots)][depths[:, :len(roots)] != 0xFFFF].max()) + 1
    assert info["push_levels"] + info["pull_levels"] == info["levels"]
    dg.close()
