"""GPU: the walk of the BF16 and FP8-B forms on the FMA engine: rows, groups
only when asked for, the same bits by both."""
from __future__ import annotations

import pytest

from graph_kernels import captured_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["bf16", "fp8_b"])
@pytest.mark.parametrize("k,n", [(512, 16), (511, 16), (512, 528), (511, 528)])
def test_groups_only_when_asked_for(native, prec, k, n):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(k + n)
    on = torch.rand(32, 128, generator=gen, device="cuda") < 0.2
    A = torch.randn(128, 512, generator=gen, device="cuda") * on.repeat_interleave(4, 0).repeat_interleave(4, 1)
    A = A[:, :k].contiguous()
    B, C = torch.randn(k, n, generator=gen, device="cuda"), torch.empty(128, n, device="cuda")
    s, out = torch.cuda.Stream(), {}
    for order, kernel in (("auto", "spdm_lowp_kernel"), ("rows", "spdm_lowp_kernel"), ("groups", "spdm_group_kernel")):
        h = native.GcooHandle(A, engine="cuda_core", fp32_order=order).build()
        h.prepare(n, prec)
        out[order] = h.spdm(B, prec=prec)
        names = [name for name, _ in captured_kernels(s, lambda: h.spdm(B, C, prec=prec, stream=s))]
        assert any(kernel in name for name in names), (order, names)
    assert torch.equal(out["auto"], out["rows"]) and torch.equal(out["auto"], out["groups"])
