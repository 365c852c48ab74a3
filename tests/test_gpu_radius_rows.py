"""Radius queries whose rows end at the sort's edges: empty, one warp's width, the shared-memory sizes, and rows long
enough for the global sort. Exact against brute force."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,leaf", [(4, 1), (8, 1), (4, 3)])
@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 63, 64, 65, 511, 512, 513, 1500])
def test_row_lengths(m, width, leaf):
    import torch
    import thea_gb300 as T
    from oracle import oracle as O
    rng = np.random.default_rng(m)
    # a cluster of m points around each of three centres, and a far query with no neighbour
    c = np.array([[0, 0, 0], [10, 0, 0], [0, 10, 0]], np.float32)
    sizes = [m, max(1, m // 2), 1]
    P = np.concatenate([c[i] + 0.1 * rng.uniform(-1, 1, size=(k, 3)) for i, k in enumerate(sizes)]).astype(np.float32)
    P = P[rng.permutation(len(P))]
    Q = np.concatenate([c, c + 0.01, [[50, 50, 50]]]).astype(np.float32)
    ex = np.array([-1, 0, -1, int(len(P)) - 1, 0, 0, -1], np.int32)
    bvh = T.PointBvh(torch.from_numpy(P).cuda(), width=width, max_leaf_size=leaf)
    off, idx, d2 = bvh.radius_neighbors(torch.from_numpy(Q).cuda(), 1.0, exclude=torch.from_numpy(ex).cuda())
    roff, ridx, rd2 = O.range_brute(P, Q, 1.0, exclude=ex)
    assert np.array_equal(off.cpu().numpy(), roff)
    assert np.array_equal(idx.cpu().numpy(), ridx)
    assert np.array_equal(d2.cpu().numpy(), rd2.astype(np.float32))
