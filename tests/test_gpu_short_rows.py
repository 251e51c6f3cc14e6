"""GPU: the short rows of skewed matrices on both sides of the number of warps
and of the long rows' length where their batches change, bit for bit against
the oracle's chains (the long rows have their own tests)."""
from __future__ import annotations

import numpy as np
import pytest

from graph_kernels import captured_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,tile", [(64, 128), (37, 32), (130, 64)])  # 4, 1 and 2 columns per lane
@pytest.mark.parametrize("longest,fp32_sum", [(600, "chain"), (2500, "chain"), (2501, "chain"), (2501, "split")])
def test_batches_by_warps_and_longest_row(native, oracle_mod, n, tile, longest, fp32_sum):
    import torch
    per_tile = 4 * 40 * torch.cuda.get_device_properties(0).multi_processor_count
    k, tiles = 2501, -(-n // tile)
    rng = np.random.default_rng(n)
    B = rng.standard_normal((k, n)).astype(np.float32)
    dB = torch.from_numpy(B).cuda()
    s, kernels = torch.cuda.Stream(), []
    for m in (per_tile // tiles, per_tile // tiles + 1):
        A = torch.zeros(m, k)
        for i, cnt in enumerate([longest, 255, 7, 8, 9, 31, 32, 33, 40, 64, 65, 0, 1, 100]):
            A[i * (m // 15), torch.from_numpy(rng.choice(k, cnt, replace=False))] = torch.from_numpy(
                rng.standard_normal(cnt).astype(np.float32))
        A[m - 1, :3] = 1.0
        filled = torch.nonzero(A.any(1))[:, 0]
        want = oracle_mod.spdm(oracle_mod.convert(A[filled].numpy()), B)
        h = native.GcooHandle(A.cuda(), fp32_sum=fp32_sum).build()
        C = h.spdm(dB)
        kernels += [name for name, _ in captured_kernels(s, lambda: h.spdm(dB, C, stream=s)) if "spdm_short" in name]
        got = C.cpu()
        assert np.array_equal(got[filled][1:].numpy().view(np.uint32), want[1:].view(np.uint32))
        bound = longest * 2.0 ** -23 * float(np.abs(A[0].numpy()) @ np.abs(B).max(1))
        assert np.allclose(got[0].numpy(), want[0], rtol=0, atol=bound)
        got[filled] = 0.0
        assert not got.any()
    # eight on the fewer warps, unless a longer chain runs beside (pieces need 16-byte copies of B)
    deep = longest <= 2500 or (fp32_sum == "split" and n % 4 == 0)
    assert len(kernels) == 2 and (kernels[0] != kernels[1]) == deep, kernels
