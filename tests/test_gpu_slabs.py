"""Oriented child slabs: built for every single-mesh BVH with the closest layout, at the sizes where the climb's runs,
warps and tree levels end, and a search that reads them finds the nearest triangle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(n, seed):
    """n random small triangles near the unit sphere; every seventh one degenerate."""
    rng = np.random.default_rng(seed)
    c = rng.normal(size=(n, 1, 3))
    c /= np.linalg.norm(c, axis=2, keepdims=True)
    t = (c + 0.05 * rng.normal(size=(n, 3, 3))).astype(np.float32)
    t[::7, 2] = t[::7, 1]
    return t.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(-1, 3)


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 255, 257, 1000, 4099])
@pytest.mark.parametrize("width,leaf", [(4, 1), (4, 2), (8, 5)])
def test_slabs_built_and_results_exact(n, width, leaf):
    import torch
    import thea_gb300 as T
    from oracle import oracle as O
    V, F = _soup(n, n)
    bvh = T.MeshBvh(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), width=width, max_leaf_size=leaf)
    inf = bvh.info()
    # nodes, both record layouts and the leaf order are counted first; the slabs take 16 bytes per child slot
    base = inf["num_nodes"] * 32 * width + n * (128 + 48 + 4)
    assert inf["device_bytes"] - base == inf["num_nodes"] * width * 16
    rng = np.random.default_rng(7)
    Q = (rng.uniform(-1, 1, size=(513, 3)) * np.array([0.2, 0.6, 1.4])[rng.integers(0, 3, size=(513, 1))])
    Q = Q.astype(np.float32)
    ri, rd2, _ = O.closest_brute(V, F, Q)
    idx, dist, _ = bvh.closest_element(torch.from_numpy(Q).cuda())
    assert np.array_equal(idx.cpu().numpy(), ri)
    assert np.array_equal(dist.cpu().numpy(), np.sqrt(rd2.astype(np.float32)))
    # the image carries no slabs: loading it builds them again
    again = T.MeshBvh.from_bytes(bvh.to_bytes())
    idx, dist, _ = again.closest_element(torch.from_numpy(Q).cuda())
    assert np.array_equal(idx.cpu().numpy(), ri)
