"""The key sort behind builds and ordered queries at its tile, tile-count and general-pass edges: a point BVH's leaf order
and k-NN graph, and FP64 re-check queries taken in Morton order, exact at every size."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 255, 256, 257, 1023, 1024, 1025, 2049, 262143, 262144, 262145])
def test_build_sorts_every_point_once(n):
    import torch
    import thea_gb300 as T
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    P = torch.rand((n, 3), generator=g, device="cuda")
    P[n // 3:n // 2] = P[0]  # equal keys
    bvh = T.PointBvh(P)
    # every point is found, at distance 0, by its own query; ties go to the lowest index
    idx, d2 = bvh.k_closest_pairs(P, 1)
    assert torch.all(d2 == 0)
    assert torch.equal(P[idx[:, 0].long()], P)
    first = torch.arange(n, device="cuda")
    first[n // 3:n // 2] = 0
    assert torch.equal(idx[:, 0].long(), first)


@pytest.mark.parametrize("n", [32768, 32769, 262144, 262145])
def test_ordered_queries(n):
    import torch
    import thea_gb300 as T
    from thea_gb300 import workloads as W
    V, F = W.noisy_icosphere(3, 4)
    bvh = T.MeshBvh(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda())
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    Q = 3 * torch.rand((n, 3), generator=g, device="cuda") - 1.5
    idx, dist, cp, _ = bvh.closest_element_ex(Q, precision="fp64", errors=False)
    for lo in (0, n // 2, n - 20000):
        i1, d1, c1, _ = bvh.closest_element_ex(Q[lo:lo + 20000].contiguous(), precision="fp64", errors=False)
        m = len(i1)
        assert torch.equal(i1, idx[lo:lo + m]) and torch.equal(d1, dist[lo:lo + m]) and torch.equal(c1, cp[lo:lo + m])
