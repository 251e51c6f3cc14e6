"""GPU: matrices dense enough for the rebuild in two passes, rows on and
off 16-byte boundaries, exact against a plain restatement of the layout."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cpg", [1, 2, 4, 8])
@pytest.mark.parametrize("m,k", [(3999, 4096), (4001, 4099), (2101, 2100), (1502, 1503)])
def test_dense_rebuilds(native, cpg, m, k):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(cpg)
    A = torch.empty(m, k, device="cuda")
    h = native.GcooHandle(A, rows_per_group=cpg)
    B = torch.ones(k, 4, device="cuda")
    for density in (0.1, 0.3, 0.5, 0.9, 0.26):  # the last build's density decides
        A.copy_(torch.randint(1, 4, (m, k), generator=gen, device="cuda"))
        A.masked_fill_(torch.rand(m, k, generator=gen, device="cuda") >= density, 0.0)
        C = h.multiply_by(B)
        assert torch.equal(C, A.sum(1, keepdim=True).expand(-1, 4))  # whole numbers: exact
        a = h.export()
        # groups in order, within a group by column, then by row
        r, c = torch.nonzero(A, as_tuple=True)
        order = torch.argsort((r // cpg) * (k * cpg) + c * cpg + r % cpg)
        assert torch.equal(a["rows"], r[order].int()) and torch.equal(a["cols"], c[order].int())
        assert torch.equal(a["vals"], A[r, c][order])
        assert h.check_arrays() == 0
