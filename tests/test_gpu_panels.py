"""GPU: the sixteen-row FP32 walk (rows of a matrix sharing columns) and the row
walk at ragged widths, bit for bit against the oracle at the edges of their
panels, windows, rings, strips and tiles."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same_bits(x, y):
    x, y = np.asarray(x, np.float32), np.asarray(y, np.float32)
    nx, ny = np.isnan(x), np.isnan(y)
    return bool(np.array_equal(nx, ny) and np.array_equal(x[~nx].view(np.uint32), y[~ny].view(np.uint32)))


def masks(rng, m, k):
    """16-row blocks; the same with a few entries missing; columns of one
    panel all full but for the ragged last one; unstructured halves."""
    blocks = np.repeat(rng.random(((m + 15) // 16, k)) < 0.3, 16, axis=0)[:m]
    holes = blocks & (rng.random((m, k)) < 0.95)
    few = np.zeros((m, k), bool)
    few[:, : min(k, 9)] = True  # one column past a ring of eight
    return {"blocks": blocks, "holes": holes, "few": few, "half": rng.random((m, k)) < 0.5}


@pytest.mark.parametrize("m,k,n", [(1, 128, 200), (16, 512, 512), (17, 516, 513), (31, 1300, 1), (48, 1024, 130),
                                   (64, 508, 129), (100, 2052, 644), (15, 4, 2048)])
def test_panels_bit_identical(native, oracle_mod, m, k, n):
    import torch
    rng = np.random.default_rng(m * 7919 + k * 31 + n)
    B = rng.standard_normal((k, n)).astype(np.float32)
    B[0, :: max(1, n // 3)] = np.inf  # only rows with an entry in column 0 may see it
    B[k // 2] = -0.0
    dB = torch.from_numpy(B).cuda()
    for name, mask in masks(rng, m, k).items():
        A = np.where(mask, rng.standard_normal((m, k)), 0.0).astype(np.float32)
        h = native.GcooHandle(torch.from_numpy(A).cuda(), fp32_order="groups").build()
        ref = oracle_mod.spdm(oracle_mod.convert(A), B)
        assert same_bits(h.spdm(dB).cpu().numpy(), ref), name
        # an unaligned C takes the 4-byte stores
        Cu = torch.empty(m * n + 1, device="cuda")[1:].view(m, n)
        assert same_bits(h.spdm(dB, Cu).cpu().numpy(), ref), name
        h.build()  # a rebuild reads A once and leaves the same prefixes
        assert same_bits(h.spdm(dB).cpu().numpy(), ref), name


@pytest.mark.parametrize("n", [64, 128, 132, 256, 320])
def test_walks_by_width_agree(native, oracle_mod, n):
    """The automatic choice changes with n (rows, groups, panels); the bits do not."""
    import torch
    from gcoospdm_gb300 import datagen as dg
    for bs in (4, 16):
        A, B = dg.block_dense(5, 96, 640, 0.3, bs=bs), dg.dense_pm1(5, 6, 640, n)
        h = native.GcooHandle(torch.from_numpy(A).cuda()).build()
        ref = oracle_mod.spdm(oracle_mod.convert(A), B)
        assert same_bits(h.spdm(torch.from_numpy(B).cuda()).cpu().numpy(), ref)


@pytest.mark.parametrize("n", [63, 65, 127, 128, 129, 191, 254, 255, 257, 258, 383, 769, 1001])
def test_ragged_widths_bit_identical(native, oracle_mod, n):
    """Widths that 16-byte (or 8-byte) loads do not fit: several narrow loads
    per lane, the last tile of a row overlapping the one before it; short
    rows (two tiles at a time), long ones, and rows beyond one staging."""
    import torch
    from gcoospdm_gb300 import datagen as dg
    for m, k, p, rows_per_group in ((37, 200, 0.02, 4), (9, 700, 0.5, 4), (5, 2600, 0.9, 8), (64, 300, 0.1, 32)):
        A, B = dg.bernoulli_dense(n, m, k, p), dg.dense_pm1(n, 6, k, n)
        C = torch.full((m + 1, n), 7.0, device="cuda")  # the row after C must stay
        h = native.GcooHandle(torch.from_numpy(A).cuda(), rows_per_group=rows_per_group, fp32_order="rows").build()
        h.spdm(torch.from_numpy(B).cuda(), C[:m])
        assert same_bits(C[:m].cpu().numpy(), oracle_mod.spdm(oracle_mod.convert(A, rows_per_group), B)), (m, k)
        assert bool((C[m] == 7.0).all())
