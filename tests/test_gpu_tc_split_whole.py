"""GPU: the split-BF16 tensor kernel on both sides of the number of tiles per
panel from which its work is cut into shares: small whole numbers, exact in
any order; ragged panels and strips, panels without entries."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(1, 16, 16), (128, 512, 128), (130, 528, 144), (1000, 500, 272), (700, 800, 400)])
@pytest.mark.parametrize("empty", [False, True])
def test_whole_panels_and_shares(native, m, k, n, empty):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    A = torch.randint(-3, 4, (m, k), generator=gen, device="cuda").float()
    A[0, 0] = 1.0
    if empty:
        A[128:384] = 0.0
    B = torch.randint(-3, 4, (k, n), generator=gen, device="cuda").float()
    panels, tiles = -(-m // 128), sum(-(-k // 16) for r in range(0, m, 128) if bool(A[r:r + 128].any()))
    h = native.GcooHandle(A, engine="tensor").build()
    h.prepare(n, "split_bf16")
    out = torch.full((m + 1, n), 7.0, device="cuda")
    L = native.lib()
    for _ in range(2):
        out[:m] = -1.0
        before = L.gcoo_kernel_launches()
        h.spdm(B, out[:m], prec="split_bf16")
        # B's tiles, the multiply and, for shares, the fix-up
        assert L.gcoo_kernel_launches() - before == (3 if tiles > 32 * panels else 2)
        assert torch.equal(out[:m], (A.double() @ B.double()).float())
        assert bool((out[m] == 7.0).all())
    assert h.device_status() == 0
