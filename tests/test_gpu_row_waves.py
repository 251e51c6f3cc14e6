"""GPU: the row walk's cut of short rows over CTAs: more of them where one row
is much longer than the others, the same bits."""
from __future__ import annotations

import numpy as np
import pytest

from graph_kernels import captured_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1600, 1601, 1602])
def test_one_longer_row(native, oracle_mod, n):
    import torch
    m, k, ctas = 3000, 500, []
    rng = np.random.default_rng(n)
    B = rng.standard_normal((k, n)).astype(np.float32)
    dB, s = torch.from_numpy(B).cuda(), torch.cuda.Stream()
    cols = np.sort(rng.integers(0, k, (m, 2)), axis=1)
    for longest in (20, 40, 200):  # a third of it below 8, below 16 and above
        A = np.zeros((m, k), np.float32)
        A[np.arange(m)[:, None], cols] = 1.5
        A[7, :longest] = rng.standard_normal(longest)
        h = native.GcooHandle(torch.from_numpy(A).cuda()).build()
        C = h.spdm(dB)
        (name, grid), = captured_kernels(s, lambda: h.spdm(dB, C, stream=s))
        assert "spdm_fp32_kernel" in name
        ctas.append(grid[0] * grid[1])
        some = np.r_[0:12, m - 4:m]
        want = oracle_mod.spdm(oracle_mod.convert(A[some]), B)
        assert np.array_equal(C.cpu().numpy()[some].view(np.uint32), want.view(np.uint32))
    assert ctas[0] < ctas[1] < ctas[2], ctas
