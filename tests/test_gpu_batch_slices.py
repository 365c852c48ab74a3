"""Mixed-precision batches longer than one slice of 16,777,216 queries: the queries on both sides of a slice's end, with a step
budget and without, answer as in calls of their own."""

import pytest

pytestmark = pytest.mark.gpu

SLICE = 1 << 24


@pytest.mark.parametrize("n", [SLICE, SLICE + 1, 2 * SLICE + 77])
def test_slices(n):
    import numpy as np
    import torch
    import thea_gb300 as T
    from thea_gb300 import workloads as W
    V0, F0 = W.noisy_icosphere(2, 4)
    V = np.concatenate([V0, V0 + [3.0, 0, 0]]).astype(np.float32)
    F = np.concatenate([F0, F0 + len(V0)]).astype(np.int32)
    forest = T.MeshForest(torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda(),
                          np.array([0, len(F0), 2 * len(F0)], np.int64))
    g = torch.Generator(device="cuda").manual_seed(n)
    Q = torch.rand((n, 3), generator=g, device="cuda") * 3 - 1.5
    half = n // 3  # queries of the first mesh
    Q[half:, 0] += 3.0
    off = torch.tensor([0, half, n], dtype=torch.int64, device="cuda")
    for budget in (-1, 0, 8):
        out = forest.batch_closest_element(Q, off, precision="fp64", hard_query_budget=budget, closest_points=True,
                                           errors=True)
        for lo, hi in ((0, 1000), (half - 300, half + 300), (SLICE - 5000, min(n, SLICE + 5000)), (n - 1000, n)):
            o = torch.tensor([0, min(max(half - lo, 0), hi - lo), hi - lo], dtype=torch.int64, device="cuda")
            ref = forest.batch_closest_element(Q[lo:hi].contiguous(), o, precision="fp64", closest_points=True, errors=True)
            for a, b in zip(out, ref):
                assert torch.equal(a[lo:hi], b)
