"""GPU: the short rows beside long rows summed in pieces, on both sides of the
number of warps where their batches change, bit for bit against the oracle's
chains (the long rows have their own tests)."""
from __future__ import annotations

import numpy as np
import pytest

from graph_kernels import captured_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,tile", [(64, 128), (37, 32), (130, 64)])  # 4, 1 and 2 columns per lane
def test_batches_by_the_number_of_warps(native, oracle_mod, n, tile):
    import torch
    per_tile = 4 * 40 * torch.cuda.get_device_properties(0).multi_processor_count
    k, tiles = 600, -(-n // tile)
    rng = np.random.default_rng(n)
    B = rng.standard_normal((k, n)).astype(np.float32)
    dB = torch.from_numpy(B).cuda()
    s, kernels = torch.cuda.Stream(), []
    for m in (per_tile // tiles, per_tile // tiles + 1):
        A = np.zeros((m, k), np.float32)
        for i, cnt in enumerate([600, 255, 7, 8, 9, 31, 32, 33, 40, 64, 65, 0, 1, 100]):
            A[i * (m // 15), rng.choice(k, cnt, replace=False)] = rng.standard_normal(cnt)
        A[m - 1, :3] = 1.0
        want = oracle_mod.spdm(oracle_mod.convert(A), B)
        C = torch.empty(m, n, device="cuda")
        h = native.GcooHandle(torch.from_numpy(A).cuda(), fp32_sum="split").build()
        C = h.spdm(dB)
        kernels += [name for name, _ in captured_kernels(s, lambda: h.spdm(dB, C, stream=s)) if "spdm_short" in name]
        assert np.array_equal(C[1:].cpu().numpy().view(np.uint32), want[1:].view(np.uint32))
        assert np.allclose(C[0].cpu().numpy(), want[0], rtol=0, atol=600 * 2.0 ** -23 * float(np.abs(A[0]) @ np.abs(B).max(1)))
    # pieces need 16-byte copies of B: other widths keep chains and batches of four
    assert len(kernels) == 2 and (kernels[0] != kernels[1]) == (n % 4 == 0), kernels
