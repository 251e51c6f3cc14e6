"""GPU: the long rows of skewed matrices, against the oracle's fmaf chains
bit by bit: lengths around the steps of both tile widths, widths around the
tiles, every alignment of B, few and many long rows (both tile widths)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [255, 256, 257, 287, 288, 289, 383, 384, 385, 512, 639, 640, 1000, 1024, 1025, 3000]


def skewed(seed, m, k, long_rows):
    rng = np.random.default_rng(seed)
    A = np.zeros((m, k), dtype=np.float32)
    for i in range(m):
        # spread over the rows, the others short or empty
        if i % (m // long_rows) == 0:
            cnt = LENGTHS[(i // (m // long_rows)) % len(LENGTHS)]
        else:
            cnt = int(rng.integers(0, 4))
        cols = rng.choice(k, size=cnt, replace=False)
        A[i, cols] = rng.standard_normal(cnt).astype(np.float32)
    return A


@pytest.mark.parametrize("m,long_rows", [(600, 16), (4800, 600)])
@pytest.mark.parametrize("n,offset", [(1, 0), (31, 0), (32, 0), (33, 0), (64, 1), (66, 2), (100, 0), (128, 0),
                                      (129, 0), (132, 2), (200, 0), (201, 3), (256, 0), (300, 1)])
def test_long_rows_bits(native, oracle_mod, m, long_rows, n, offset):
    import torch
    k = 3000
    A = skewed(m + n, m, k, long_rows)
    B = np.random.default_rng(n).standard_normal((k, n)).astype(np.float32)
    want = oracle_mod.spdm(oracle_mod.convert(A), B)
    buf = torch.zeros(k * n + 4, device="cuda")
    dB = buf[offset:offset + k * n].view(k, n)
    dB.copy_(torch.from_numpy(B))
    out = torch.full((m + 1, n), 7.0, device="cuda")
    h = native.GcooHandle(torch.from_numpy(A).cuda()).build()
    for _ in range(2):
        out[:m] = -1.0
        h.spdm(dB, out[:m])
        assert np.array_equal(out[:m].cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert bool((out[m] == 7.0).all())
    assert h.device_status() == 0
