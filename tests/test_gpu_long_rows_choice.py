"""GPU: when the long and short rows of a skewed matrix get kernels of their
own and when its rows or panels are walked, the same bits either way."""
from __future__ import annotations

import pytest

from graph_kernels import captured_kernels

pytestmark = pytest.mark.gpu


# few long rows at little work; nearly all rows long and one four times as
# long; the same at unaligned widths; blocks of 16 rows beside one full row
@pytest.mark.parametrize("kind,n,kernel", [
    ("few", 64, "spdm_long_kernel"), ("few", 65, "spdm_long_kernel"), ("few", 66, "spdm_long_kernel"),
    ("few", 2001, "spdm_fp32_kernel"),
    ("all", 64, "spdm_long_kernel"), ("all", 1024, "spdm_fp32_kernel"), ("all", 1023, "spdm_fp32_kernel"),
    ("all", 33, "spdm_fp32_kernel"), ("blocks", 64, "spdm_long_kernel"), ("blocks", 2048, "spdm_panel_kernel")])
def test_kernels_by_work(native, kind, n, kernel):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    m, k = 4992, 4096
    density = {"few": 0.01, "all": 0.11, "blocks": 0.1}[kind]
    if kind == "blocks":
        on = torch.rand(m // 16, k // 16, generator=gen, device="cuda") < density
        on = on.repeat_interleave(16, 0).repeat_interleave(16, 1)
    else:
        on = torch.rand(m, k, generator=gen, device="cuda") < density
    A = torch.randn(m, k, generator=gen, device="cuda") * on
    A[5] = torch.randn(k, generator=gen, device="cuda")
    B = torch.randn(k, n, generator=gen, device="cuda")
    h = native.GcooHandle(A).build()
    C, s = h.spdm(B), torch.cuda.Stream()
    want = C.clone()
    names = [name for name, _ in captured_kernels(s, lambda: h.spdm(B, C, stream=s))]
    assert any(kernel in name for name in names), names
    for order in ("rows", "groups"):
        assert torch.equal(want, native.GcooHandle(A, fp32_order=order).build().spdm(B)), order
