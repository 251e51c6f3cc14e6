"""GPU: the caller-array entry points (count, scatter, multiply from arrays in
the reference layout) at the edges of their chunks, tiles and groups, exact
against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cpg", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("m,k,n,density", [(37, 200, 1, 0.02), (33, 515, 65, 0.3), (64, 2050, 129, 0.02),
                                           (5, 2600, 256, 0.9), (100, 129, 1001, 0.1), (16, 4096, 130, 0.5),
                                           (3, 7, 33, 0.0)])
def test_caller_arrays(native, oracle_mod, m, k, n, density, cpg):
    import torch
    rng = np.random.default_rng(m + k + n)
    A = np.where(rng.random((m, k)) < density, rng.standard_normal((m, k)), 0.0).astype(np.float32)
    if density:
        A[0, 0] = A[m - 1, k - 1] = 2.0
    B = rng.standard_normal((k, n)).astype(np.float32)
    ref = oracle_mod.convert(A, cpg)
    want = oracle_mod.spdm(ref, B).view(np.uint32)
    buf = torch.full((m * k + 8,), 9.0, device="cuda")
    dB = torch.from_numpy(B).cuda()
    for shift in (0, 1, 2):
        dA = buf[shift:shift + m * k].view(m, k)
        dA.copy_(torch.from_numpy(A))
        gi, npg, nnz = native.convert_count(dA, cpg)
        assert nnz == ref.vals.size
        vals, rows, cols = native.convert_scatter(dA, gi, nnz, cpg)
        for got, field in ((gi, "groupIndex"), (npg, "nnzPerGroup"), (rows, "rows"), (cols, "cols")):
            assert np.array_equal(got.cpu().numpy(), getattr(ref, field)), field
        assert np.array_equal(vals.cpu().numpy().view(np.uint32), ref.vals.view(np.uint32))
        C = torch.full((m + 1, n), 7.0, device="cuda")
        native.spdm_view(m, k, cpg, gi, npg, vals, rows, cols, dB, C[:m])
        assert np.array_equal(C[:m].cpu().numpy().view(np.uint32), want)
        assert bool((C[m] == 7.0).all())


def test_view_skips_rows_of_other_groups(native, oracle_mod):
    """Entries whose row is not in their group take no part (and break nothing)."""
    import torch
    rng = np.random.default_rng(5)
    A = np.where(rng.random((24, 90)) < 0.2, rng.standard_normal((24, 90)), 0.0).astype(np.float32)
    B = rng.standard_normal((90, 77)).astype(np.float32)
    ref = oracle_mod.convert(A, 4)
    rows = ref.rows.copy()
    at = ref.groupIndex[2]  # the first entry of group 2
    A2 = A.copy()
    A2[rows[at], ref.cols[at]] = 0.0
    rows[at] = 0
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    C = native.spdm_view(24, 90, 4, t(ref.groupIndex), t(ref.nnzPerGroup), t(ref.vals), t(rows), t(ref.cols), t(B))
    want = oracle_mod.spdm(oracle_mod.convert(A2, 4), B)
    assert np.array_equal(C.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("cpg", [1, 2, 4])
@pytest.mark.parametrize("n", [1, 55, 130, 256])
def test_groups_around_a_chunk(native, oracle_mod, n, cpg):
    """Groups of one entry less and more than one, two and three staged chunks (256 entries per row of a group)."""
    import torch
    rng = np.random.default_rng(n + cpg)
    totals = [c * 256 * cpg + d for c in (1, 2, 3) for d in (-1, 0, 1)] + [0, 1]
    k = 800
    A = np.zeros((len(totals) * cpg, k), np.float32)
    for i, total in enumerate(totals):
        at = rng.choice(cpg * k, total, replace=False)
        A[i * cpg + at // k, at % k] = rng.standard_normal(total)
    B = rng.standard_normal((k, n)).astype(np.float32)
    ref = oracle_mod.convert(A, cpg)
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    C = native.spdm_view(A.shape[0], k, cpg, t(ref.groupIndex), t(ref.nnzPerGroup), t(ref.vals), t(ref.rows),
                         t(ref.cols), t(B))
    assert np.array_equal(C.cpu().numpy().view(np.uint32), oracle_mod.spdm(ref, B).view(np.uint32))


@pytest.mark.parametrize("cpg", [1, 4, 8, 16])
@pytest.mark.parametrize("m,entries", [(3000, 1), (40000, 1), (40000, 7), (3000, 9), (700, 17)])
def test_short_rows(native, cpg, m, entries):
    """Rows of few entries, few and many waves of groups: one strip of columns per group or several."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + entries)
    k = 300
    A = torch.randint(1, 5, (m, k), generator=gen, device="cuda").float()
    A.masked_fill_(torch.rand(m, k, generator=gen, device="cuda") >= entries / k, 0.0)
    gi, npg, nnz = native.convert_count(A, cpg)
    vals, rows, cols = native.convert_scatter(A, gi, nnz, cpg)
    for n in (1, 130, 801):
        B = torch.randint(-8, 9, (k, n), generator=gen, device="cuda").float()
        C = torch.full((m + 1, n), 7.0, device="cuda")
        native.spdm_view(m, k, cpg, gi, npg, vals, rows, cols, B, C[:m])
        want = native.GcooHandle(A, fp32_order="rows").build().spdm(B)
        assert torch.equal(C[:m], want) and bool((C[m] == 7.0).all())
        assert torch.equal(want.double(), A.double() @ B.double())  # whole numbers: exact
