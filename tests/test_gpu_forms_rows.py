"""GPU: the reduced-precision row walk (FMA engine) at the edges of its tiles,
batches and staged chunks, bit for bit against the FP32 chain over the rounded
operands (split-BF16: within FP32 rounding of the exact product)."""
from __future__ import annotations

import numpy as np
import pytest

from fp8_emu import e4m3_round, fp8_scales

pytestmark = pytest.mark.gpu


def bf16(x):
    u = np.ascontiguousarray(x, np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) & np.uint32(0xFFFF0000)).view(np.float32)


@pytest.mark.parametrize("n", [16, 256, 272, 512, 1008, 1024, 1040, 2064])
@pytest.mark.parametrize("m,k,density,cpg", [(9, 300, 0.03, 4), (6, 700, 0.6, 2), (5, 2600, 0.9, 4), (3, 40, 0.0, 1)])
def test_row_walk(native, oracle_mod, m, k, density, cpg, n):
    import torch
    rng = np.random.default_rng(m + k + n)
    A = np.where(rng.random((m, k)) < density, rng.uniform(-1, 1, (m, k)), 0.0).astype(np.float32)
    B = rng.uniform(-1, 1, (k, n)).astype(np.float32) * np.exp2(rng.integers(-3, 4, n)).astype(np.float32)
    h = native.GcooHandle(torch.from_numpy(A).cuda(), rows_per_group=cpg, engine="cuda_core", fp32_order="rows").build()
    dB = torch.from_numpy(B).cuda()

    def same(got, want):
        return np.array_equal(got.cpu().numpy().view(np.uint32), want.astype(np.float32).view(np.uint32))

    assert same(h.spdm(dB, prec="bf16"), oracle_mod.spdm(oracle_mod.convert(bf16(A), cpg), bf16(B)))
    scale = fp8_scales(B)
    assert same(h.spdm(dB, prec="fp8_b"), oracle_mod.spdm(oracle_mod.convert(A, cpg), e4m3_round(B / scale)) * scale)
    C = h.spdm(dB, prec="split_bf16").cpu().numpy().astype(np.float64)
    exact = A.astype(np.float64) @ B.astype(np.float64)
    # two BF16 terms keep a and b to 2^-18 each and al * bl, at most 2^-18, is
    # left out: below 2^-16 of each product; and three FP32 roundings per entry
    bound = (2.0 ** -16 + 3 * k * 2.0 ** -24) * (np.abs(A).astype(np.float64) @ np.abs(B).astype(np.float64))
    assert bool((np.abs(C - exact) <= bound).all())


def test_prepared_width_serves_smaller_ones_in_a_capture(native):
    """gcoo_prepare at one width: every smaller width multiplies without an
    allocation (which a capture would refuse), whichever format of B it reads."""
    import torch
    from gcoospdm_gb300 import datagen as dg
    A = dg.bernoulli_dense_torch(3, 64, 500, 0.1, device="cuda")
    h = native.GcooHandle(A, engine="cuda_core").build()
    h.prepare(2048, "fp8_b")
    s = torch.cuda.Stream()
    for n in (2048, 1040, 1024, 256):
        B = dg.dense_pm1_torch(4, 5, 500, n, device="cuda")
        C = torch.empty(64, n, device="cuda")
        graph = torch.cuda.CUDAGraph()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.graph(graph, stream=s):
            h.spdm(B, C, prec="fp8_b", stream=s)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(C, h.spdm(B, prec="fp8_b"))
