"""breadthFirstSearchGraphCSR's host results on both sides of the size at which
they take another way to the host (65536 vertices), of searches shorter and
longer than 255 levels: depths exact, parents valid."""
import ctypes as C

import numpy as np
import pytest

from test_bfs_gpu import check_parents

pytestmark = pytest.mark.gpu


def edges(V, kind):
    rng = np.random.default_rng(V)
    if kind == "chain":
        s = np.arange(V - 1)
        d = s + 1
    else:
        s, d = rng.integers(0, V, (2, 8 * V))
        s[0] = V - 1  # an edge file's vertex count is its largest id + 1
    return s.astype(np.uint32), d.astype(np.uint32)


@pytest.mark.parametrize("V,kind", [(2, "chain"), (300, "chain"), (1000, "uniform"), (65535, "uniform"),
                                    (65536, "uniform"), (65537, "uniform"), (65536, "chain")])
def test_results(og, lib, oracle, tmp_path, V, kind):
    s, d = edges(V, kind)
    path = str(tmp_path / "g.bin")
    og.write_edge_file(path, s, d)
    args = og.default_arguments(fnameb=path, sort=0, pushpull=2)
    lib.initializeMersenneState(C.byref(args.mt19937var), 27491095)
    h = lib.graphCSRPreProcessingStep(C.byref(args))
    g = oracle.build(s, d, V, 0)
    for root in (0, V // 2):
        if g["f_outdeg"][root] == 0:
            continue
        args.source = root
        for _ in range(2):  # the second call's arrays are the first's, recycled
            st = lib.breadthFirstSearchGraphCSR(C.byref(args), h)
            r = st.contents
            par, dist = og.as_numpy(r.parents, V, np.int32), og.as_numpy(r.distances, V, np.uint32)
            _, edist, est = oracle.bfs(g, root, 2)
            assert np.array_equal(dist, edist)
            assert r.processed_nodes == est["processed_nodes"] and r.iteration == est["iteration"]
            check_parents(g, root, par, dist)
            lib.freeBFSStats(st)
    lib.graphCSRFree(h)
