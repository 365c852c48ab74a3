"""Queries with infinite coordinates in the mixed-precision mode: whichever kernel finishes them (a thread, a warp from the
root, the collecting kernel and a warp after it), they find the same element, at infinite distance."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,leaf", [(4, 1), (4, 5), (8, 2)])
@pytest.mark.parametrize("level", [3, 5])
def test_infinite_queries(level, width, leaf):
    import torch
    import thea_gb300 as T
    from thea_gb300 import workloads as W
    V, F = W.noisy_icosphere(level, 3)
    Vd, Fd = torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda()
    bvh = T.MeshBvh(Vd, Fd, width=width, max_leaf_size=leaf)
    forest = T.MeshForest(Vd, Fd, np.array([0, len(F)], np.int64), width=width, max_leaf_size=leaf)
    Q = W.uniform_box_points(4000, [-1.5] * 3, [1.5] * 3, 2)
    Q[7] = np.inf
    Q[8, 2] = -np.inf
    Q[9, 1] = np.nan
    Qd = torch.from_numpy(Q).cuda()
    ref = None
    for n in (10, 2047, 2500, 4000):
        idx, dist, _, _ = bvh.closest_element_ex(Qd[:n].contiguous(), precision="fp64")
        if ref is None:
            ref = idx[7:10].tolist()
            assert ref[0] >= 0 and ref[1] >= 0 and ref[2] == -1
        assert idx[7:10].tolist() == ref
        assert torch.all(torch.isinf(dist[7:9])) and dist[9] == -1
    off = torch.tensor([0, len(Q)], dtype=torch.int64, device="cuda")
    for budget in (-1, 0, 1, 64):
        idx, dist = forest.batch_closest_element(Qd, off, precision="fp64", hard_query_budget=budget)[:2]
        assert idx[7:10].tolist() == ref
        assert torch.all(torch.isinf(dist[7:9])) and dist[9] == -1
