"""GPU: the tiled conversion where A's rows do not start on 16 bytes (odd k,
views into a larger buffer), first builds and one-read rebuilds, exact against
the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(h, ref):
    a = h.export()
    assert a["nnz"] == ref.vals.size
    for name in ("groupIndex", "nnzPerGroup", "rows", "cols"):
        assert np.array_equal(a[name].cpu().numpy(), getattr(ref, name)), name
    assert np.array_equal(a["vals"].cpu().numpy().view(np.uint32), ref.vals.view(np.uint32))
    assert h.check_arrays() == 0
    assert h.device_status() == 0


@pytest.mark.parametrize("cpg", [1, 2, 4, 8])
@pytest.mark.parametrize("k", [1, 2, 3, 5, 127, 129, 1023, 1024, 1025, 1027, 2050, 4099])
def test_ragged_rows_convert(native, oracle_mod, k, cpg):
    import torch
    rng = np.random.default_rng(k * 8 + cpg)
    m = 13
    A = np.where(rng.random((m, k)) < 0.05, rng.standard_normal((m, k)), 0.0).astype(np.float32)
    A[:cpg, : min(k, 1024)] = 1.5  # one tile that overflows its slot on rebuilds
    A[m - 1, k - 1] = -2.0  # the very last element, and the first
    A[0, 0] = 3.0
    ref = oracle_mod.convert(A, cpg)
    for shift in range(4):
        # A inside a larger buffer whose other floats are nonzero: none of them may appear
        buf = torch.full((m * k + 8,), 9.0, device="cuda")
        view = buf[shift:shift + m * k].view(m, k)
        view.copy_(torch.from_numpy(A))
        h = native.GcooHandle(view, rows_per_group=cpg).build()
        check(h, ref)
        h.build()
        check(h, ref)
        view[m // 2].zero_()
        A2 = A.copy()
        A2[m // 2] = 0.0
        h.build()
        check(h, oracle_mod.convert(A2, cpg))


@pytest.mark.parametrize("cpg", [4, 8])
@pytest.mark.parametrize("m", [1, 31, 33, 8192, 8193, 16384, 16385])
def test_row_scan_edges(native, oracle_mod, m, cpg):
    """The one-launch prefix and scan (up to 16384 rows, 32 rows per CTA, 8192
    per scan chunk) and the launches beyond it; first build, rebuild, and a
    multiply that goes ahead of the rebuild's readback, also where the arrays
    turn out too small for it."""
    import torch
    rng = np.random.default_rng(m + cpg)
    A = np.where(rng.random((m, 130)) < 0.1, rng.standard_normal((m, 130)), 0.0).astype(np.float32)
    B = rng.standard_normal((130, 36)).astype(np.float32)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    h = native.GcooHandle(dA, rows_per_group=cpg).build()
    check(h, oracle_mod.convert(A, cpg))
    for density in (0.1, 0.02, 0.9, 0.9):
        A = np.where(rng.random((m, 130)) < density, rng.standard_normal((m, 130)), 0.0).astype(np.float32)
        dA.copy_(torch.from_numpy(A))
        C = h.multiply_by(dB)
        ref = oracle_mod.convert(A, cpg)
        check(h, ref)
        assert np.array_equal(C.cpu().numpy().view(np.uint32), oracle_mod.spdm(ref, B).view(np.uint32))
