"""Closest point of small batches (32 and 16 lanes per query): batch sizes at the ends of the teams, warps and blocks and
on both sides of the switch, queries deep inside, near and outside the surface, with and without a distance bound, and
against the persistent kernels' answer for the same queries."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _queries(n, seed):
    rng = np.random.default_rng(seed)
    q = rng.normal(size=(n, 3))
    q *= (rng.choice([0.0, 0.3, 1.0, 1.6], size=(n, 1)) + 0.02 * rng.normal(size=(n, 1))) / np.linalg.norm(
        q, axis=1, keepdims=True)
    return q.astype(np.float32)


@pytest.mark.parametrize("width,leaf", [(4, 1), (4, 2), (4, 7), (8, 2)])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 15, 17, 3071, 3072, 3073, 9001])
def test_small_batches(n, width, leaf):
    import torch
    import thea_gb300 as T
    from oracle import oracle as O
    from thea_gb300 import workloads as W
    V, F = W.noisy_icosphere(3, 5)
    bvh = T.MeshBvh(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), width=width, max_leaf_size=leaf)
    Q = _queries(n, n)
    for bound in (-1.0, 0.25):
        idx, dist, cp = bvh.closest_element(torch.from_numpy(Q).cuda(), bound)
        ri, rd2, rcp = O.closest_brute(V, F, Q, dist_bound=bound)
        found = ri >= 0
        assert np.array_equal(idx.cpu().numpy(), ri)
        assert np.array_equal(dist.cpu().numpy()[found], np.sqrt(rd2[found].astype(np.float32)))
        assert np.all(dist.cpu().numpy()[~found] == -1)
        assert np.array_equal(cp.cpu().numpy()[found], rcp.astype(np.float32)[found])


def test_same_answers_as_the_large_batch():
    import torch
    import thea_gb300 as T
    from thea_gb300 import workloads as W
    V, F = W.noisy_icosphere(6, 6)
    bvh = T.MeshBvh(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda())
    Q = torch.from_numpy(_queries(100000, 7)).cuda()
    ref = bvh.closest_element(Q)
    for lo, hi in ((0, 1000), (1000, 4100), (5000, 60000)):
        got = bvh.closest_element(Q[lo:hi].contiguous())
        for a, b in zip(got, ref):
            assert torch.equal(a, b[lo:hi])
    nan = Q[:40].clone()
    nan[3, 1] = float("nan")
    nan[4] = float("inf")
    idx, dist, _ = bvh.closest_element(nan)
    keep = torch.ones(40, dtype=torch.bool, device="cuda")
    keep[3:5] = False
    assert torch.equal(idx[keep], ref[0][:40][keep])
    assert int(idx[3]) == -1 and float(dist[3]) == -1.0
