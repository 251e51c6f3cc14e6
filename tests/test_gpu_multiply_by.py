"""GPU: multiply_by on a handle whose matrix changes its nature between calls
(the multiply may be enqueued before the new totals are known), and on one
whose conversion fails."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def natures(rng, m, k):
    even = rng.random((m, k)) < 0.02
    skewed = rng.random((m, k)) < 0.002
    skewed[:: m // 8, : k // 2] = True
    block = np.repeat(np.repeat(rng.random((m // 16, k // 16)) < 0.3, 16, 0), 16, 1)
    low = np.repeat(np.repeat(rng.random((m // 4, k // 4)) < 0.3, 4, 0), 4, 1)
    return {"even": even, "skewed": skewed, "block": block, "low": low, "empty": np.zeros((m, k), bool)}


@pytest.mark.parametrize("n", [64, 320, 130])
@pytest.mark.parametrize("rows_per_group", [4, 8])
def test_changing_matrices(native, oracle_mod, n, rows_per_group):
    """Every change from one kind of matrix to another, bit for bit."""
    import torch
    m, k = 256, 2048
    rng = np.random.default_rng(n)
    B = rng.standard_normal((k, n)).astype(np.float32)
    dB, dA = torch.from_numpy(B).cuda(), torch.zeros(m, k, device="cuda")
    h = native.GcooHandle(dA, rows_per_group=rows_per_group)
    kinds = {}
    for name, mask in natures(rng, m, k).items():
        A = np.where(mask, rng.standard_normal((m, k)), 0.0).astype(np.float32)
        ref = oracle_mod.convert(A, rows_per_group)
        kinds[name] = torch.from_numpy(A).cuda(), ref, oracle_mod.spdm(ref, B)
    C = torch.full((m + 1, n), 7.0, device="cuda")
    for first in kinds:
        for second in kinds:
            for name in (first, second):
                A, ref, want = kinds[name]
                dA.copy_(A)
                C[:m] = -1.0
                h.multiply_by(dB, C[:m])
                assert np.array_equal(C[:m].cpu().numpy().view(np.uint32), want.view(np.uint32)), (first, second)
                assert bool((C[m] == 7.0).all())
            assert h.check_arrays() == 0 and h.nnz == ref.vals.size
            again = h.spdm(dB).cpu().numpy()  # by whichever walk the new totals chose
            assert np.array_equal(again.view(np.uint32), want.view(np.uint32)), (first, second)
    assert h.device_status() == 0


def test_failed_conversion_leaves_c(native):
    """More nonzeros than the int32 format holds, found by a rebuild with the
    multiply enqueued behind it: an error, and C as it was."""
    import torch
    m = k = 46400  # 46400^2 > 2^31
    A = torch.zeros(m, k, device="cuda")
    A.diagonal().fill_(1.0)
    B, C = torch.ones(k, 4, device="cuda"), torch.full((m, 4), 7.0, device="cuda")
    h = native.GcooHandle(A)
    h.multiply_by(B, C)
    h.multiply_by(B, C)
    assert bool((C == 1.0).all())
    A.fill_(1.0)
    C.fill_(7.0)
    with pytest.raises(native.GcooError) as e:
        h.multiply_by(B, C)
    assert "int32" in str(e.value)
    torch.cuda.synchronize()
    assert bool((C == 7.0).all())
    A.zero_()
    A.diagonal().fill_(2.0)
    h.multiply_by(B, C)  # and the handle goes on
    torch.cuda.synchronize()
    assert bool((C == 2.0).all())
