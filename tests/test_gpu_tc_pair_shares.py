"""GPU: the pair kernel (BF16, FP8-B) where its work is cut into shares that
reach over strips of columns and over several panels: parts of a strip other
than the first, whole panels inside a share, a tensor-memory bank's second
piece. Small whole numbers: exact in any order."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one panel of 1250 tiles in two strips, in three with a ragged last one; 154
# panels of 64 tiles in shares of 130, each the end of a panel, a whole one and
# the start of a third; 40 panels of 512 tiles, two of them empty, in four strips
@pytest.mark.parametrize("m,k,n,density", [(200, 20000, 512, 1.0), (130, 20000, 528, 1.0), (39424, 1024, 16, 1.0),
                                           (10230, 8192, 1024, 0.9)])
@pytest.mark.parametrize("prec", ["bf16", "fp8_b"])
def test_shares_over_strips_and_panels(native, m, k, n, density, prec):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    A = torch.randint(-3, 4, (m, k), generator=gen, device="cuda").float()
    if density < 1.0:
        on = torch.rand((m + 15) // 16, k // 16, generator=gen, device="cuda") < density
        A *= on.repeat_interleave(16, 0)[:m].repeat_interleave(16, 1)
        A[512:1024] = 0.0  # two panels without entries
    B = torch.randint(-3, 4, (k, n), generator=gen, device="cuda").float()
    B[0] = 3.0  # every column's absmax: a power-of-two scale keeps the numbers in E4M3
    want = (A.double() @ B.double()).float()
    h = native.GcooHandle(A, engine="tensor").build()
    h.prepare(n, prec)
    out = torch.full((m + 1, n), 7.0, device="cuda")
    L = native.lib()
    for _ in range(2):
        out[:m] = -1.0
        before = L.gcoo_kernel_launches()
        h.spdm(B, out[:m], prec=prec)
        # B's tiles, the multiply and the fix-up that only shares need (FP8-B: the scales' two as well)
        assert L.gcoo_kernel_launches() - before == (3 if prec == "bf16" else 5)
        assert torch.equal(out[:m], want)
        assert bool((out[m] == 7.0).all())
    assert h.device_status() == 0


@pytest.mark.parametrize("m,k,n", [(206, 4980, 192), (112, 2807, 480), (439, 2934, 112)])
def test_few_panels_of_few_tiles_stay_whole(native, m, k, n):
    """A share of four tiles each, seventy to be added per panel: not cut."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m)
    A = torch.randint(-3, 4, (m, k), generator=gen, device="cuda").float()
    B = torch.randint(-3, 4, (k, n), generator=gen, device="cuda").float()
    h = native.GcooHandle(A, engine="tensor").build()
    h.prepare(n, "bf16")
    L = native.lib()
    before = L.gcoo_kernel_launches()
    C = h.spdm(B, prec="bf16")
    assert L.gcoo_kernel_launches() - before == 2  # B's tiles and the multiply
    assert torch.equal(C, (A.double() @ B.double()).float())
