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
    in a wide matrix they lie; a rebuild chooses as the first build. (Asked
    for either: by themselves so few rows take the row walk.)"""
    import torch
    A = blocks(64, 1 << 18, bs, 0.06, first_col)
    h = native.GcooHandle(A, fp32_order="groups").build()
    B, C = torch.ones(1 << 18, 1024, device="cuda"), torch.empty(64, 1024, device="cuda")
    s = torch.cuda.Stream()
    for _ in range(2):
        names = [name for name, _ in captured_kernels(s, lambda: h.spdm(B, C, stream=s))]
        assert len(names) == 1 and kernel in names[0], names
        h.build()
        torch.cuda.synchronize()


@pytest.mark.parametrize("rows,holes,n,kernel", [
    (2, 0.0, 1024, "spdm_fp32_kernel"), (2, 0.0, 1001, "spdm_fp32_kernel"), (2, 0.0, 128, "spdm_fp32_kernel"),
    (4, 0.0, 1024, "spdm_group_kernel"), (4, 0.0, 1001, "spdm_fp32_kernel"), (4, 0.0, 512, "spdm_fp32_kernel"),
    (16, 0.4, 2048, "spdm_panel_kernel"), (16, 0.4, 2001, "spdm_fp32_kernel"), (16, 0.4, 1024, "spdm_fp32_kernel"),
    (16, 0.0, 1001, "spdm_panel_kernel")])
@pytest.mark.parametrize("k", [2048, 2047])
def test_choice_by_sharing_and_work(native, rows, holes, n, kernel, k):
    """Blocks of several heights at 15 %: the walk by how many rows share a
    column and by the work, whatever the rows' alignment; the same bits by
    every walk."""
    import torch
    A = blocks(2048, 2048, rows, 0.15)[:, :k].contiguous()
    A *= torch.rand(2048, k, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda") >= holes
    h = native.GcooHandle(A).build()
    gen = torch.Generator(device="cuda").manual_seed(3)
    B, C = torch.randn(k, n, generator=gen, device="cuda"), torch.empty(2048, n, device="cuda")
    s = torch.cuda.Stream()
    names = [name for name, _ in captured_kernels(s, lambda: h.spdm(B, C, stream=s))]
    assert len(names) == 1 and kernel in names[0], names
    want = h.spdm(B, C).clone()
    for order in ("rows", "groups"):
        assert torch.equal(want, native.GcooHandle(A, fp32_order=order).build().spdm(B)), order


@pytest.mark.parametrize("m,k,density,n,kernel", [
    (2048, 2048, 0.25, 256, "spdm_panel_kernel"),  # four windows of 512 columns
    (2048, 16384, 0.03125, 256, "spdm_fp32_kernel"),  # as many entries in 32
    (2048, 16384, 0.25, 256, "spdm_panel_kernel")])  # long rows
def test_choice_by_the_windows(native, m, k, density, n, kernel):
    """Few entries in each of many windows of columns: not the panels."""
    import torch
    A = blocks(m, k, 16, density)
    h = native.GcooHandle(A).build()
    B, C = torch.ones(k, n, device="cuda"), torch.empty(m, n, device="cuda")
    s = torch.cuda.Stream()
    names = [name for name, _ in captured_kernels(s, lambda: h.spdm(B, C, stream=s))]
    assert len(names) == 1 and kernel in names[0], names
    torch.cuda.synchronize()
    assert torch.equal(h.spdm(B), A.sum(1, keepdim=True).expand(-1, n))  # whole numbers: exact


@pytest.mark.parametrize("bs,kernel", [(16, "spdm_panel_kernel"), (2, "spdm_fp32_kernel")])
@pytest.mark.parametrize("m,k", [(2048, 2047), (2047, 2050), (4096, 4096)])
def test_choice_of_dense_rebuilds(native, m, k, bs, kernel):
    """Matrices so dense that a rebuild reads A twice: the sample of A itself
    tells what that of the first build's entries told, also when the matrix
    has turned to other blocks in between."""
    import torch
    blk = lambda bs: blocks(2048 if m < 4000 else m, 4096, bs, 0.5)[:m, :k].contiguous()  # noqa: E731
    A = blk(bs)
    h = native.GcooHandle(A).build()
    B, C = torch.ones(k, 256, device="cuda"), torch.empty(m, 256, device="cuda")
    s = torch.cuda.Stream()
    for turn in range(3):
        names = [name for name, _ in captured_kernels(s, lambda: h.spdm(B, C, stream=s))]
        assert len(names) == 1 and kernel in names[0], (turn, names)
        torch.cuda.synchronize()
        assert torch.equal(h.spdm(B), A.sum(1, keepdim=True).expand(-1, 256))  # whole numbers: exact
        if turn == 0:
            A.copy_(blk(18 - bs))
            h.build()
            A.copy_(blk(bs))
        h.build()


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
