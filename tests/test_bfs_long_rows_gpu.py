"""Bottom-up steps over long in-rows: rows around the lengths at which a row
goes from four lanes to a warp and from a warp to the CTA, whose first frontier
in-neighbour is early, late or absent, and more such rows than a round hands on.
Pull-only searches take the first frontier in-neighbour in CSR order, so their
parents are compared too."""
import numpy as np
import pytest

from test_bfs_gpu import check_parents
from test_build_gpu import dev, host

pytestmark = pytest.mark.gpu


def graph(lengths, V, seed):
    """Root 0 -> 1..200; vertex 1000 + i has lengths[i] in-edges from vertices
    the root does not reach, and, two times in three, one from 1..200 at a random
    place of the row (rows are sorted by source id, so the ids are permuted)."""
    rng = np.random.default_rng(seed)
    far = np.arange(V // 2, V)
    ss, dd = [np.zeros(200, np.int64)], [np.arange(1, 201)]
    for i, n in enumerate(lengths):
        s = rng.choice(far, size=n)
        if i % 3:
            s = np.append(s, rng.integers(1, 201))
        ss.append(s)
        dd.append(np.full(len(s), 1000 + i))
    s, d = np.concatenate(ss), np.concatenate(dd)
    perm = rng.permutation(V)
    order = rng.permutation(len(s))
    return perm[s][order].astype(np.uint32), perm[d][order].astype(np.uint32), int(perm[0])


def examined(g, root, par, dist, steps):
    """Edges read by `steps` bottom-up steps: in every step each unvisited
    vertex's row up to its first in-neighbour of the step's frontier."""
    reached = par >= 0
    total = 0
    for depth in range(1, steps + 1):
        frontier = reached & (dist == depth - 1)
        for v in np.nonzero((g["i_outdeg"] > 0) & ~(reached & (dist < depth)))[0]:
            if v == root:
                continue
            row = g["i_dst"][g["i_idx"][v]: g["i_idx"][v] + g["i_outdeg"][v]]
            hit = np.nonzero(frontier[row])[0]
            total += int(hit[0]) + 1 if len(hit) else len(row)
    return total


ROWS = {
    "edges": [3, 4, 5, 67, 68, 69, 70, 71, 72, 76, 195, 196, 197, 2111, 2112, 2113, 2116, 3135, 3140, 9000, 30_001] * 3,
    "many": [120] * 3000,          # more rows than a round hands to the warps
    "hubs": [2500] * 400,          # more rows than a round hands to the CTA
}


@pytest.mark.parametrize("name", list(ROWS))
def test_long_rows(torch_cuda, lib, oracle, name):
    torch = torch_cuda
    V = 8192
    s, d, root = graph(ROWS[name], V, 7)
    g = oracle.build(s, d, V, 0)
    dg = lib.device_graph()
    dg.build(dev(torch, s), dev(torch, d), V, 0)
    par_t = torch.empty(V, dtype=torch.int32, device="cuda")
    dist_t = torch.empty(V, dtype=torch.int32, device="cuda")
    for mode in (0, 2, 4):  # 4: pull with every step over all vertices
        info = dg.bfs(root, par_t, dist_t, mode=mode)
        epar, edist, est = oracle.bfs(g, root, 0 if mode == 4 else mode)
        par, dist = host(par_t, np.int32), host(dist_t)
        assert np.array_equal(dist, edist), mode
        for k in ("iteration", "processed_nodes", "reached", "reached_out_edges"):
            assert info[k] == est[k], (mode, k)
        check_parents(g, root, par, dist)
        if mode != 2:
            assert np.array_equal(par, epar), mode
            assert info["edges_examined"] == examined(g, root, par, dist, info["bu_steps"]), mode
    dg.close()
