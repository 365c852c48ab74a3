"""k nearest points at the edges of the lists: every capacity and rows shorter than it, fewer points than k, duplicate
points, exclusions, bounds that admit nothing, sizes around the self mode's starting window, and small batches that use
one lane of a warp or all of them. Bit-exact against brute force."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(n, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(-1, 1, size=(n, 3)).astype(np.float32)
    p[n // 2:n // 2 + n // 8] = p[:n // 8]  # duplicates: ties in distance
    return p


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 7, 8, 9, 12, 15, 16, 17, 20, 31, 32])
@pytest.mark.parametrize("n,width,leaf", [(1, 4, 1), (2, 4, 1), (9, 4, 2), (33, 8, 1), (700, 4, 1), (701, 4, 5)])
def test_lists(k, n, width, leaf):
    import torch
    import thea_gb300 as T
    from oracle import oracle as O
    P = _points(n, n)
    bvh = T.PointBvh(torch.from_numpy(P).cuda(), width=width, max_leaf_size=leaf)
    idx, d2 = bvh.k_closest_self(k, device=True)
    ri, rd = O.knn_brute(P, P, k, exclude=np.arange(n, dtype=np.int32))
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(d2.cpu().numpy(), rd.astype(np.float32))
    rng = np.random.default_rng(k)
    Q = np.concatenate([rng.uniform(-1.5, 1.5, size=(200, 3)).astype(np.float32), P[:57]])
    ex = np.where(np.arange(len(Q)) % 3 == 0, rng.integers(0, n, size=len(Q)), -1).astype(np.int32)
    for bound in (-1.0, 0.0, 0.3):
        idx, d2 = bvh.k_closest_pairs(torch.from_numpy(Q).cuda(), k, bound, torch.from_numpy(ex).cuda())
        ri, rd = O.knn_brute(P, Q, k, dist_bound=bound, exclude=ex)
        assert np.array_equal(idx.cpu().numpy(), ri)
        assert np.array_equal(d2.cpu().numpy(), rd.astype(np.float32))


@pytest.mark.parametrize("n", [1, 33, 3647, 3649, 7297, 58369, 116737])
def test_batches_of_every_density(n):
    """One to 32 queries a warp (the steps lie at multiples of 24 x 152 warps), against single calls of other density."""
    import torch
    import thea_gb300 as T
    P = torch.from_numpy(_points(5000, 1)).cuda()
    bvh = T.PointBvh(P)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    Q = 2 * torch.rand((n, 3), generator=g, device="cuda") - 1
    idx, d2 = bvh.k_closest_pairs(Q, 8)
    off, ri, rd = bvh.radius_neighbors(Q, 0.1)
    for lo in range(0, n, max(1, n // 3)):
        hi = min(n, lo + 500)
        i1, e1 = bvh.k_closest_pairs(Q[lo:hi].contiguous(), 8)
        assert torch.equal(i1, idx[lo:hi]) and torch.equal(e1, d2[lo:hi])
        o1, r1, f1 = bvh.radius_neighbors(Q[lo:hi].contiguous(), 0.1)
        a, b = int(off[lo]), int(off[hi])
        assert torch.equal(o1 + off[lo], off[lo:hi + 1]) and torch.equal(r1, ri[a:b]) and torch.equal(f1, rd[a:b])
