"""Batched k-NN on both sides of the batch sizes from which lists are kept sorted in shared memory: each row equals the same
query's in a smaller call (the other form of list), with every distance bound, with ties, and with fewer points in a set than
neighbours asked for."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bound", [-1.0, 0.0, 0.2, float("inf"), float("nan")])
@pytest.mark.parametrize("width,k,n", [(4, 17, 98304), (4, 32, 98304), (8, 32, 98304), (8, 16, 524288), (8, 9, 524288)])
def test_sorted_lists(width, k, n, bound):
    import torch
    import thea_gb300 as T
    g = torch.Generator(device="cuda").manual_seed(k)
    sets, per = 8, 500
    P = torch.rand((sets * per + 5, 3), generator=g, device="cuda")
    P[per:2 * per] = (P[per:2 * per] * 8).round() / 8  # ties
    off = list(range(0, sets * per + 1, per)) + [sets * per + 5]  # the last set has five points
    import numpy as np
    forest = T.PointForest(P, np.array(off, np.int64), width=width)
    Q = torch.rand((n, 3), generator=g, device="cuda")
    Q[1] = float("nan")
    Q[2, 0] = float("inf")
    m = len(off) - 1
    qoff = torch.linspace(0, n, m + 1, device="cuda").round().to(torch.int64)
    idx, d2 = forest.batch_k_closest(Q, qoff, k, bound)
    for s in range(m):  # each set's queries in a call of their own
        lo, hi = int(qoff[s]), int(qoff[s + 1])
        own = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
        own[s + 1:] = hi - lo
        ri, rd = forest.batch_k_closest(Q[lo:hi].contiguous(), own, k, bound)
        assert torch.equal(idx[lo:hi], ri) and torch.equal(d2[lo:hi], rd)
