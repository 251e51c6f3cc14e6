"""GPU: the row walk's launch shapes by rows per group and by how many CTAs
there are for the GPU's SMs, bit for bit against the oracle on some rows."""
from __future__ import annotations

import numpy as np
import pytest

from graph_kernels import captured_kernels

pytestmark = pytest.mark.gpu


def check(native, oracle_mod, m, k, n, per_row, rows_per_group=4):
    import torch
    rng = np.random.default_rng(m + n)
    A = np.where(rng.random((m, k)) < per_row / k, rng.standard_normal((m, k)), 0.0).astype(np.float32)
    B = rng.standard_normal((k, n)).astype(np.float32)
    h = native.GcooHandle(torch.from_numpy(A).cuda(), rows_per_group=rows_per_group, fp32_order="rows").build()
    C = torch.full((m + 1, n), 7.0, device="cuda")
    dB, s = torch.from_numpy(B).cuda(), torch.cuda.Stream()
    for _ in range(3):  # one behind another
        h.spdm(dB, C[:m])
    some = np.r_[0:9, m // 2, m - 5:m]
    want = oracle_mod.spdm(oracle_mod.convert(A[some]), B)
    assert np.array_equal(C.cpu().numpy()[some].view(np.uint32), want.view(np.uint32))
    assert bool((C[m] == 7.0).all()) and bool((C[:m] != 7.0).any(1).all())
    (name, grid), = captured_kernels(s, lambda: h.spdm(dB, C[:m], stream=s))
    return name, grid[0] * grid[1]


@pytest.mark.parametrize("rows_per_group", [8, 16, 32])
@pytest.mark.parametrize("per_row", [7, 130])
@pytest.mark.parametrize("n", [100, 133, 518])
def test_many_rows_per_group(native, oracle_mod, rows_per_group, per_row, n):
    check(native, oracle_mod, 1003, 400, n, per_row, rows_per_group)


@pytest.mark.parametrize("n", [128, 131, 258, 512])
def test_one_wave_of_ten_and_of_twelve_ctas(native, oracle_mod, n):
    """Around 10 and 12 CTAs per SM: twelve are resident only in the kernel of fewer registers."""
    import torch
    sms, names = torch.cuda.get_device_properties(0).multi_processor_count, []
    tiles = -(-n // 128)
    for per_sm in (9.9, 10.1, 11.9, 12.1):
        name, ctas = check(native, oracle_mod, 4 * int(per_sm * sms / tiles), 300, n, 140)
        assert abs(ctas - per_sm * sms) <= tiles
        names.append(name)
    assert names[0] == names[3] != names[1] == names[2], names


@pytest.mark.parametrize("rows_per_group", [1, 4, 8, 32])
@pytest.mark.parametrize("n", [1, 100, 133])
def test_rows_longer_than_a_chunk(native, oracle_mod, rows_per_group, n):
    """Rows of more entries than a CTA stages at once: one row per CTA."""
    m = 301
    _, ctas = check(native, oracle_mod, m, 2700, n, 2400, rows_per_group)
    assert ctas % m == 0, ctas
