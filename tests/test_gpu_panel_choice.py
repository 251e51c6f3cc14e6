"""GPU: how a build learns whether sixteen rows share their columns: by what
evidence, and without holding up a multiply that is already under way."""
from __future__ import annotations

import pytest

from graph_kernels import captured_kernels

pytestmark = pytest.mark.gpu


def blocks(m, k, bs, density, first_col=0, seed=1):
    """bs x bs blocks from first_col on, on the GPU."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    on = torch.rand(m // bs, (k - first_col) // bs, generator=gen, device="cuda") < density
    A = torch.zeros(m, k, device="cuda")
    A[:, first_col:] = on.repeat_interleave(bs, 0).repeat_interleave(bs, 1)
    return A


@pytest.mark.parametrize("bs,first_col,kernel", [(16, 0, "spdm_panel_kernel"), (4, 0, "spdm_group_kernel"),
                                                 (16, 1 << 17, "spdm_panel_kernel"), (4, 1 << 17, "spdm_group_kernel")])
def test_choice_by_the_blocks_height(native, bs, first_col, kernel):
    """Blocks as high as a panel take the panels, lower ones do not, wherever
    in a wide matrix they lie; a rebuild chooses as the first build."""
    import torch
    A = blocks(64, 1 << 18, bs, 0.1, first_col)
    h = native.GcooHandle(A).build()
    B, C = torch.ones(1 << 18, 320, device="cuda"), torch.empty(64, 320, device="cuda")
    s = torch.cuda.Stream()
    for _ in range(2):
        names = [name for name, _ in captured_kernels(s, lambda: h.spdm(B, C, stream=s))]
        assert len(names) == 1 and kernel in names[0], names
        h.build()
        torch.cuda.synchronize()


@pytest.mark.parametrize("m,k,rows,n,kernel", [
    (2048, 2048, 2, 320, "spdm_panel_kernel"), (2048, 2048, 2, 1024, "spdm_fp32_kernel"),
    (2048, 2048, 8, 1024, "spdm_panel_kernel"), (2048, 8192, 2, 1024, "spdm_group_kernel"),
    (2048, 2048, 2, 1001, "spdm_panel_kernel"), (2048, 2048, 2, 128, "spdm_fp32_kernel")])
def test_choice_by_the_gain(native, m, k, rows, n, kernel):
    """Blocks of two rows at 15 %, half of the columns shared by a group's rows
    and few more by a panel's: the panels where they gain enough on the
    groups, the same bits by every walk."""
    import torch
    A = blocks(m, k, rows, 0.15)
    if rows == 8:
        A *= torch.rand(m, k, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda") < 0.6
    h = native.GcooHandle(A).build()
    gen = torch.Generator(device="cuda").manual_seed(3)
    B, C = torch.randn(k, n, generator=gen, device="cuda"), torch.empty(m, n, device="cuda")
    s = torch.cuda.Stream()
    names = [name for name, _ in captured_kernels(s, lambda: h.spdm(B, C, stream=s))]
    assert len(names) == 1 and kernel in names[0], names
    assert torch.equal(h.spdm(B, C), native.GcooHandle(A, fp32_order="rows").build().spdm(B))


def test_multiply_by_returns_with_the_multiply_under_way(native):
    """A steady loop on a block matrix whose width takes the row walk (here
    milliseconds of it): the call waits for the conversion's totals only."""
    import torch
    A = blocks(65536, 8192, 16, 0.05)
    B, C = torch.ones(8192, 128, device="cuda"), torch.empty(65536, 128, device="cuda")
    h = native.GcooHandle(A)
    h.multiply_by(B, C)
    s = torch.cuda.current_stream()
    running = []
    for _ in range(4):
        torch.cuda.synchronize()
        h.multiply_by(B, C)
        running.append(not s.query())
    torch.cuda.synchronize()
    assert sum(running) >= 3, running
    assert torch.equal(C, A.sum(1, keepdim=True).expand(-1, 128))  # whole numbers: exact
