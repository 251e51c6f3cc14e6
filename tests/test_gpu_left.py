"""GPU: the other orientation (C = D x A) at the edges of its transposes'
tiles and of their 16-byte accesses, bit for bit against the chain over A's
rows in ascending order."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,p", [(1, 1, 1), (63, 65, 3), (64, 64, 64), (65, 130, 4), (128, 67, 129), (66, 260, 63),
                                   (100, 33, 260)])
def test_left(native, oracle_mod, m, k, p):
    import torch
    rng = np.random.default_rng(m + k + p)
    A = np.where(rng.random((m, k)) < 0.2, rng.standard_normal((m, k)), 0.0).astype(np.float32)
    D = rng.standard_normal((p, m)).astype(np.float32)
    # C^T = A^T x D^T, each element a chain over A's rows
    want = oracle_mod.spdm(oracle_mod.convert(np.ascontiguousarray(A.T)), np.ascontiguousarray(D.T)).T
    h = native.GcooHandle(torch.from_numpy(A).cuda()).build()
    for shift in (0, 1):  # an unaligned D and C take the 4-byte accesses
        buf, out = torch.empty(p * m + 1, device="cuda"), torch.full((p * k + 2,), 7.0, device="cuda")
        dD, C = buf[shift:shift + p * m].view(p, m), out[shift:shift + p * k].view(p, k)
        dD.copy_(torch.from_numpy(D))
        h.spdm_left(dD, C)
        assert np.array_equal(C.cpu().numpy().view(np.uint32), np.ascontiguousarray(want).view(np.uint32))
        assert float(out[shift + p * k]) == 7.0
