"""When a search hands its narrow steps to the cluster kernel: paths with hubs
every few vertices, counted in launches (the search kernel once, and twice more
per run).  Runs too short to pay must not be tried again and again, long ones must
go on, a long one lets short lists start a run again, and a frontier that grows or
shrinks fast starts none."""
import numpy as np
import pytest

from test_bfs_gpu import check_parents
from test_bfs_narrow_gpu import layered
from test_build_gpu import dev, host

pytestmark = pytest.mark.gpu


def hub_path(sections):
    """A path; a section is (length, period, leaves): every period-th of its
    vertices, its first among them, has that many leaves (period 0: none)."""
    hubs, at = [], 0
    for length, period, leaves in sections:
        if period:
            hubs += [(v, leaves) for v in range(at, at + length, period)]
        at += length
    ls = np.concatenate([np.full(k, v) for v, k in hubs] + [np.zeros(0, np.int64)]).astype(np.int64)
    s = np.concatenate([np.arange(at - 1), ls])
    d = np.concatenate([np.arange(1, at), at + np.arange(len(ls))])
    V = at + len(ls)
    perm = np.random.default_rng(3).permutation(V)
    return perm[s].astype(np.uint32), perm[d].astype(np.uint32), V, int(perm[0])


# a run starts after 4, then 8, ... narrow lists of about equal length; the two after a hub's are not
CASES = {
    "every5": ([(1000, 5, 33)], 1),               # 4 such lists in a row never come
    "every8": ([(1000, 8, 1000)], 3),             # a run of 2 steps; 8 lists never come
    "every12": ([(1200, 12, 33)], 5),             # 6 steps, then 2
    "every15": ([(1500, 15, 100)], 1 + 2 * 100),  # 9 steps: as good either way, and it stays
    "every100": ([(1000, 100, 40)], 1 + 2 * 10),
    "none": ([(600, 0, 0)], 3),
    "reset": ([(500, 8, 33), (500, 0, 0), (500, 8, 33)], 1 + 2 * 3),
}
# layers of these widths
LAYERS = {
    "even": ([1, 4, 16, 64] + [700] * 30, 4, 3),
    "doubling": ([1 << k for k in range(15)], 2, 3),
    "tripling": ([3 ** k for k in range(10)], 3, 1),
    "shrinking": ([1, 32, 1000, 20_000, 1500, 400, 100, 25, 6], 32, 1),
}


NO_CLUSTERS = 2  # test option of a graph: as on a device that cannot launch the cluster


@pytest.mark.parametrize("clusters", [True, False])
@pytest.mark.parametrize("name", list(CASES) + list(LAYERS))
def test_launches(torch_cuda, lib, oracle, name, clusters):
    torch = torch_cuda
    if name in CASES:
        sections, launches = CASES[name]
        s, d, V, root = hub_path(sections)
    else:
        widths, degree, launches = LAYERS[name]
        s, d, V, root = layered(widths, degree, 3)
    g = oracle.build(s, d, V, 0)
    dg = lib.device_graph()
    if not clusters:
        launches = 1
        lib.check(lib.ogb_graph_test_option(dg.handle, NO_CLUSTERS, 1))
    dg.build(dev(torch, s), dev(torch, d), V, 0)
    par_t = torch.empty(V, dtype=torch.int32, device="cuda")
    dist_t = torch.empty(V, dtype=torch.int32, device="cuda")
    for _ in range(2):  # the second search starts anew
        info = dg.bfs(root, par_t, dist_t, mode=1)
        _, edist, est = oracle.bfs(g, root, 1)
        assert np.array_equal(host(dist_t), edist)
        for k in ("iteration", "processed_nodes", "td_steps", "reached", "reached_out_edges"):
            assert info[k] == est[k], k
        check_parents(g, root, host(par_t, np.int32), host(dist_t))
        assert info["launches"] == launches
    dg.close()
