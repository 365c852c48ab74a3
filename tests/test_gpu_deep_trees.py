"""Trees far deeper than a balanced one, whose every node keeps most of its children within the search's bound: the searches
that finish a query with a whole warp hold their node stack within its bounds and answer as on any other tree."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEVELS = 60


def nested_mesh(per, slope):
    """Eight octants whose triangles converge on the origin: at each of LEVELS binary splits, the half away from it holds
    `per` triangles. Their boxes overlap (a box is far larger than its cell): deeper ones reach nearer to a query on the +x
    side, shallower ones have the larger area (the collapse opens them first, so that a wide node's inner child is one
    split deeper), and none of the triangles themselves comes near it."""
    V = []
    for octant in range(8):
        s = np.array([1 if octant & 4 else -1, 1 if octant & 2 else -1, 1 if octant & 1 else -1], float)
        ext = np.ones(3)
        for i in range(LEVELS):
            a, b, d = i % 3, (i + 1) % 3, (i + 2) % 3
            c = np.where(np.arange(3) == a, 0.75 * ext, 0.5 * ext)
            hx, hy = 4.0 + 0.02 * i, 64 + slope * (LEVELS - i)
            for k in range(per):
                off = np.zeros(3)
                off[b] = (0.25 if k & 1 else -0.25) * ext[b]
                off[d] = (0.25 if k & 2 else -0.25) * ext[d]
                off[a] = (0.06 if k & 4 else -0.06) * ext[a]
                u = -1 if (k + i) & 1 else 1
                v = -1 if (k // 2 + i) & 1 else 1
                V.append(s * (c + off) + np.array([[hx, u * hy, v * hy], [-hx, -u * hy, v * hy], [-hx, u * hy, -v * hy]]))
            ext[a] *= 0.5
    V = np.concatenate(V).astype(np.float32)
    return V, np.arange(len(V), dtype=np.int32).reshape(-1, 3)


def queries(n):
    rng = np.random.default_rng(n)
    return (np.array([20.0, 0.0, 0.0]) + 0.01 * rng.normal(size=(n, 3))).astype(np.float32)


@pytest.mark.parametrize("width,per", [(4, 12), (8, 32)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_deep_trees(width, per, precision):
    import torch
    import thea_gb300 as T
    from oracle import oracle as O
    V, F = nested_mesh(per, 2.0)
    Vd, Fd = torch.from_numpy(V).cuda(), torch.from_numpy(F).cuda()
    bvh = T.MeshBvh(Vd, Fd, width=width, max_leaf_size=1)
    assert bvh.info()["depth"] > 45  # the warp's stack would have to hold (32 / width) ((width - 1) depth + 1) entries
    Q = queries(4000)
    ri, rd2, _ = O.closest_brute(V, F, Q[:200], fp64=precision == "fp64")
    rd = np.sqrt(rd2) if precision == "fp64" else np.sqrt(rd2.astype(np.float32))
    forest = T.MeshForest(Vd, Fd, np.array([0, len(F)], np.int64), width=width, max_leaf_size=1)
    off = torch.tensor([0, len(Q)], dtype=torch.int64, device="cuda")
    Qd = torch.from_numpy(Q).cuda()
    for got in (bvh.closest_element_ex(Qd, precision=precision, errors=False),
                forest.batch_closest_element(Qd, off, precision=precision, hard_query_budget=1),
                forest.batch_closest_element(Qd, off, precision=precision)):
        assert np.array_equal(got[0].cpu().numpy()[:200], ri)
        assert np.all(np.abs(got[1].cpu().numpy()[:200] - rd) <= 2.0 ** -23 * rd)
    assert bvh.info()["device_error_bits"] == 0
    assert forest.info()["device_error_bits"] == 0
