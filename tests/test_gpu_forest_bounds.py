"""Distance-bounded batches over forests: each mesh's bound (and the cut of its own root box) applies to its queries alone,
so a batch answers as closestElement on each mesh does."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("meshes", [1, 5, 1500])
def test_bounded_batches(meshes, precision):
    import torch
    import thea_gb300 as T
    from thea_gb300 import workloads as W
    V0, F0 = W.noisy_icosphere(1, 4)
    rng = np.random.default_rng(meshes)
    scale = rng.uniform(0.5, 2.0, (meshes, 1, 1))
    shift = rng.uniform(-3.0, 3.0, (meshes, 1, 3))
    V = (V0[None] * scale + shift).astype(np.float32)
    F = (F0[None] + len(V0) * np.arange(meshes)[:, None, None]).reshape(-1, 3).astype(np.int32)
    forest = T.MeshForest(torch.from_numpy(V.reshape(-1, 3)).cuda(), torch.from_numpy(F).cuda(),
                          np.arange(meshes + 1, dtype=np.int64) * len(F0))
    per = 24
    Q = (rng.normal(size=(meshes, per, 3)) * scale * 1.2 + shift).astype(np.float32)
    off = torch.arange(meshes + 1, dtype=torch.int64, device="cuda") * per
    for bound in (0.05, 0.4, 5.0):
        idx, dist = forest.batch_closest_element(torch.from_numpy(Q.reshape(-1, 3)).cuda(), off, bound,
                                                 precision=precision)[:2]
        idx, dist = idx.cpu().numpy().reshape(meshes, per), dist.cpu().numpy().reshape(meshes, per)
        seen = set()
        for m in sorted({0, meshes // 2, meshes - 1} | set(range(0, meshes, 100))):
            one = T.MeshBvh(torch.from_numpy(V[m]).cuda(), torch.from_numpy(F0.astype(np.int32)).cuda())
            ri, rd = one.closest_element_ex(torch.from_numpy(Q[m]).cuda(), bound, precision=precision)[:2]
            assert np.array_equal(idx[m], ri.cpu().numpy())
            assert np.array_equal(dist[m], rd.cpu().numpy())
            seen |= set((idx[m] >= 0).tolist())
        assert meshes == 1 or bound == 5.0 or seen == {False, True}
