"""GPU: the tensor engine's cut of the work into shares: small integers, whose
FP32 sums are exact in any order, so every element has to be exact whatever
the panels, widths and shares are (empty panels, fewer tiles than one share,
panels in many shares, ragged edges)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["split_bf16", "bf16", "fp8_b"])
@pytest.mark.parametrize("m,k,n,density", [(1, 5, 16, 1.0), (128, 16, 16, 1.0), (300, 2000, 144, 0.3),
                                           (1000, 4096, 16, 0.2), (2048, 256, 400, 0.1), (130, 20000, 32, 0.05),
                                           (520, 640, 1040, 0.5), (257, 1024, 272, 0.4)])
def test_integer_products_exact(native, m, k, n, density, prec):
    import torch
    rng = np.random.default_rng(m + k + n)
    mask = rng.random(((m + 15) // 16, (k + 15) // 16)) < density
    A = rng.integers(-3, 4, (m, k)) * np.repeat(np.repeat(mask, 16, 0)[:m], 16, 1)[:, :k]
    if m > 600:
        A[256:512] = 0  # panels without entries
    if not A.any():
        A[0, 0] = 1
    B = rng.integers(-3, 4, (k, n))
    B[0] = 3  # every column's absmax: a power-of-two scale keeps the integers in E4M3
    want = (A @ B).astype(np.float32)
    h = native.GcooHandle(torch.from_numpy(A.astype(np.float32)).cuda(), engine="tensor").build()
    out = torch.full((m + 1, n), 7.0, device="cuda")
    dB = torch.from_numpy(B.astype(np.float32)).cuda()
    for _ in range(2):  # twice: nothing of the first run's parts may be left over
        out[:m] = -1.0
        h.spdm(dB, out[:m], prec=prec)
        assert np.array_equal(out[:m].cpu().numpy(), want)
        assert bool((out[m] == 7.0).all())
    assert h.device_status() == 0
