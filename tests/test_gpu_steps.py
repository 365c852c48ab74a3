"""The searches' shared step loads: leaves of every size (a leaf's records start at even and odd places, end at the
array's end, and come one or two to a step), widths 4 and 8, in the one-per-thread and the persistent-lane kernels, and
stacks deeper than their shared-memory part. Bit-exact against the brute-force oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(n, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 1, size=(n, 1, 3))
    t = (c + 0.1 * rng.normal(size=(n, 3, 3))).astype(np.float32)
    return t.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(-1, 3)


def _tiled(a, n):
    """a repeated up to n rows (the persistent kernels need large batches; the oracle does not)."""
    return np.concatenate([a] * (n // len(a) + 1))[:n]


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("n,leaf", [(1, 1), (2, 2), (3, 2), (5, 3), (17, 16), (33, 5), (1000, 1), (1001, 2), (999, 16)])
def test_leaves_of_every_size(n, leaf, width):
    import torch
    import thea_gb300 as T
    from oracle import oracle as O
    V, F = _soup(n, 31 * n + leaf)
    bvh = T.MeshBvh(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), width=width, max_leaf_size=leaf)
    rng = np.random.default_rng(3)
    o = rng.uniform(-1, 2, size=(601, 3)).astype(np.float32)
    d = (rng.uniform(0, 1, size=(601, 3)) - o).astype(np.float32)
    rt, ri = O.ray_brute(V, F, o, d)
    ci, cd2, _ = O.closest_brute(V, F, o)
    for m in (601, 70001):
        to, td = torch.from_numpy(_tiled(o, m)).cuda(), torch.from_numpy(_tiled(d, m)).cuda()
        t, idx, _ = bvh.ray_structure_intersection(to, td)
        assert np.array_equal(idx.cpu().numpy(), _tiled(ri, m))
        assert np.array_equal(t.cpu().numpy(), _tiled(rt.astype(np.float32), m))
        hit = bvh.ray_intersects(to, td)
        assert np.array_equal(hit.cpu().numpy(), _tiled(ri, m) >= 0)
    for m in (601, 60001, 100001):
        idx, dist, _ = bvh.closest_element(torch.from_numpy(_tiled(o, m)).cuda())
        assert np.array_equal(idx.cpu().numpy(), _tiled(ci, m))
        assert np.array_equal(dist.cpu().numpy(), _tiled(np.sqrt(cd2.astype(np.float32)), m))


def test_image_keeps_the_last_records_readable():
    import torch
    import thea_gb300 as T
    V, F = _soup(4097, 5)
    bvh = T.MeshBvh(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda())
    again = T.MeshBvh.from_bytes(bvh.to_bytes())
    rng = np.random.default_rng(4)
    o = torch.from_numpy(rng.uniform(-1, 2, size=(70001, 3)).astype(np.float32)).cuda()
    d = torch.rand_like(o) - o
    for a, b in zip(bvh.ray_structure_intersection(o, d)[:2], again.ray_structure_intersection(o, d)[:2]):
        assert torch.equal(a, b)
