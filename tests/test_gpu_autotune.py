"""The autotuner on a sample whose size the library's own default step budget is 256 for: that budget is among the candidates,
so the choice is not slower than a call that names none."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_sample():
    import torch
    import thea_gb300 as T
    from thea_gb300 import workloads as W
    V0, F0 = W.noisy_icosphere(2, 4)
    M, per = 16, 6144
    V = np.concatenate([V0 + [3.0 * m, 0, 0] for m in range(M)]).astype(np.float32)
    F = np.concatenate([F0 + len(V0) * m for m in range(M)]).astype(np.int32)
    off = np.arange(M + 1, dtype=np.int64) * len(F0)
    Q = np.concatenate([W.uniform_box_points(per, [-1.5] * 3, [1.5] * 3, m) + np.float32([3.0 * m, 0, 0])
                        for m in range(M)]).astype(np.float32)
    qoff = torch.arange(M + 1, dtype=torch.int64, device="cuda") * per
    dev = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    for n, candidates in ((M * per, 48), (M * per - 1, 36)):
        qo = qoff.clone()
        qo[-1] = n
        tune = T.autotune_batch_closest(dev(V), dev(F), off, dev(Q[:n]), qo)
        assert tune["candidates"] == candidates
        assert tune["hard_query_budget"] in (12, 32, 128, 256, 384, -1)
