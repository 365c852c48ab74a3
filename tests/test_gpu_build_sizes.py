"""Builds on both sides of the size from which nodes are counted before they are written, at both widths: the nearest points
of a sample of queries against brute force, and the tree's own account of its elements."""

import pytest

pytestmark = pytest.mark.gpu

LINE = 1 << 21


@pytest.mark.parametrize("width,leaf", [(4, 1), (8, 1), (4, 5)])
@pytest.mark.parametrize("n", [262145, LINE, LINE + 1, 2 * LINE + 7])
def test_sizes(n, width, leaf):
    import torch
    import thea_gb300 as T
    g = torch.Generator(device="cuda").manual_seed(n)
    P = torch.rand((n, 3), generator=g, device="cuda")
    P[: n // 2] *= 0.01  # half of them in a corner: uneven subtrees
    bvh = T.PointBvh(P, width=width, max_leaf_size=leaf)
    Q = torch.cat([P[:64] + 1e-4, P[-64:] + 1e-3])
    idx, d2 = bvh.k_closest_pairs(Q, 3)
    for i in range(len(Q)):
        d = ((P - Q[i]) ** 2)
        d = d[:, 0] + (d[:, 1] + d[:, 2])
        ref, _ = torch.sort(d)
        got = ((P[idx[i].long()] - Q[i]) ** 2)
        got = got[:, 0] + (got[:, 1] + got[:, 2])
        assert torch.allclose(got, ref[:3], rtol=3e-7, atol=0)
        assert torch.allclose(d2[i], ref[:3], rtol=3e-7, atol=0)
    info = bvh.info()
    assert info["num_elements"] == n and info["device_error_bits"] == 0
