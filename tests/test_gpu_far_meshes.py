"""Closest point on meshes far from the origin (coordinates hundreds of times their size): the bounds that the searches prune
by are taken from large coordinates whose products nearly cancel. Every size rule's kernel, against the oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("offset", [30.0, 1000.0])
def test_far_mesh(offset, precision):
    import torch
    import thea_gb300 as T
    from oracle import oracle as O
    from thea_gb300 import workloads as W
    V, F = W.noisy_icosphere(4, 3)
    at = offset * np.array([1.0, -0.7, 0.4])
    V = (V + at).astype(np.float32)
    bvh = T.MeshBvh(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda())
    rng = np.random.default_rng(7)
    Q = rng.normal(size=(100003, 3))
    Q *= rng.choice([0.2, 1.0, 1.5], size=(len(Q), 1)) / np.linalg.norm(Q, axis=1, keepdims=True)
    Q = (Q + at).astype(np.float32)
    ri, rd2, _ = O.closest_brute(V, F, Q[:300], fp64=precision == "fp64")
    for n in (300, 5000, 60000, 100003):
        idx, dist, _, _ = bvh.closest_element_ex(torch.from_numpy(Q[:n]).cuda(), precision=precision, errors=False)
        assert np.array_equal(idx.cpu().numpy()[:300], ri)
        if precision == "fp32":
            assert np.array_equal(dist.cpu().numpy()[:300], np.sqrt(rd2.astype(np.float32)))
