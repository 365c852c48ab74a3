"""The key sort behind builds where it changes from its two-launch form to the general pass: 160 tiles of 1,024 keys. Every
point is found once, ties by index, on both sides."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [160 * 1024 - 1, 160 * 1024, 160 * 1024 + 1])
def test_switch(n):
    import torch
    import thea_gb300 as T
    g = torch.Generator(device="cuda").manual_seed(n)
    P = torch.rand((n, 3), generator=g, device="cuda")
    P[n // 3:n // 2] = P[0]  # equal keys
    idx, d2 = T.PointBvh(P).k_closest_pairs(P, 1)
    first = torch.arange(n, device="cuda")
    first[n // 3:n // 2] = 0
    assert torch.all(d2 == 0)
    assert torch.equal(idx[:, 0].long(), first)
