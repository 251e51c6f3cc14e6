"""GPU: counting and scattering into a caller's arrays, A's rows on and off
16-byte boundaries, exact against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cpg", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("k", [4, 1023, 1024, 1025, 2050])
@pytest.mark.parametrize("density", [0.05, 0.6])
def test_scatter_into_own_arrays(native, oracle_mod, cpg, k, density):
    import torch
    rng = np.random.default_rng(cpg + k)
    m = 37
    A = np.where(rng.random((m, k)) < density, rng.standard_normal((m, k)), 0.0).astype(np.float32)
    A[0, 0], A[m - 1, k - 1] = 3.0, -2.0
    ref = oracle_mod.convert(A, cpg)
    for shift in range(4):
        # inside a larger buffer whose other floats are nonzero: none of them may appear
        buf = torch.full((m * k + 8,), 9.0, device="cuda")
        view = buf[shift:shift + m * k].view(m, k)
        view.copy_(torch.from_numpy(A))
        index, per_group, nnz = native.convert_count(view, cpg)
        vals, rows, cols = native.convert_scatter(view, index, nnz, cpg)
        assert nnz == ref.vals.size
        for got, want in ((index, ref.groupIndex), (per_group, ref.nnzPerGroup), (rows, ref.rows), (cols, ref.cols)):
            assert np.array_equal(got.cpu().numpy(), want)
        assert np.array_equal(vals.cpu().numpy().view(np.uint32), ref.vals.view(np.uint32))
