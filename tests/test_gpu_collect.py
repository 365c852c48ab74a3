"""The mixed-precision search's collecting and resolving kernels: more band entries than a lane keeps (many triangles at one
distance), queries handed to the warp-per-query kernel by the step budget, meshes on both sides of the small-mesh rule and
batches on both sides of each size rule, with distance bounds and error estimates. Indices equal the FP64 oracle's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(bvh, V, F, Q, bound, oracle_q):
    import torch
    from oracle import oracle as O
    idx, dist, cp, err = bvh.closest_element_ex(torch.from_numpy(Q).cuda(), bound, precision="fp64")
    pick = np.linspace(0, len(Q) - 1, min(len(Q), oracle_q)).astype(np.int64)
    ri, rd2, rcp = O.closest_brute(V, F, Q[pick], dist_bound=bound, fp64=True)
    got = idx.cpu().numpy()[pick]
    assert np.array_equal(got, ri)
    found = ri >= 0
    rd = np.sqrt(rd2[found])
    # the FP64 distance rounded to FP32
    assert np.all(np.abs(dist.cpu().numpy()[pick][found] - rd) <= 2.0 ** -23 * rd + 1e-30)
    assert np.all(err.cpu().numpy()[pick][found] <= 2.0 ** -23 * np.maximum(rd, 1e-30))
    assert np.all(dist.cpu().numpy()[pick][~found] == -1)


@pytest.mark.parametrize("bound", [-1.0, 0.2])
@pytest.mark.parametrize("level", [3, 4])
@pytest.mark.parametrize("n", [1, 3071, 3073, 8191, 8193, 32769, 40001])
def test_sizes(n, level, bound):
    import torch
    import thea_gb300 as T
    from thea_gb300 import workloads as W
    V, F = W.noisy_icosphere(level, 3)
    bvh = T.MeshBvh(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda())
    Q = W.uniform_box_points(n, [-1.5] * 3, [1.5] * 3, n)
    _check(bvh, V, F, Q, bound, 400)


@pytest.mark.parametrize("leaf", [1, 2, 9])
@pytest.mark.parametrize("width", [4, 8])
def test_many_band_entries(width, leaf):
    """A fan of triangles around a vertex: a query above it has every one of them at the same distance."""
    import torch
    import thea_gb300 as T
    m = 3000
    a = np.linspace(0, 2 * np.pi, m, endpoint=False)
    rim = np.stack([np.cos(a), np.sin(a), -0.5 + 0 * a], 1)
    V = np.concatenate([[[0, 0, 0]], rim]).astype(np.float32)
    F = np.stack([np.zeros(m), 1 + np.arange(m), 1 + (np.arange(m) + 1) % m], 1).astype(np.int32)
    bvh = T.MeshBvh(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), width=width, max_leaf_size=leaf)
    rng = np.random.default_rng(2)
    Q = (rng.normal(size=(5000, 3)) * 0.01 + [0, 0, 1]).astype(np.float32)
    _check(bvh, V, F, Q, -1.0, 300)


@pytest.mark.parametrize("width,leaf", [(4, 7), (4, 8), (4, 15), (8, 8)])
@pytest.mark.parametrize("n", [32767, 32768])
def test_leaf_sizes_at_the_budget_rule(n, width, leaf):
    """Either side of the larger step budget of leaves of eight, queries around and deep inside the mesh."""
    import torch
    import thea_gb300 as T
    from thea_gb300 import workloads as W
    V, F = W.noisy_icosphere(5, 3)
    bvh = T.MeshBvh(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(), width=width, max_leaf_size=leaf)
    _check(bvh, V, F, W.uniform_box_points(n, [-1.5] * 3, [1.5] * 3, n), -1.0, 200)
