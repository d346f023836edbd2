"""AMG refresh with every level factored on a stream of its own, and the one-pass level defects."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


def _grid(n):
    """5-point pattern of an n x n grid, sorted CSR."""
    t = sp.diags([1, 1, 1], [-1, 0, 1], shape=(n, n))
    a = (sp.kron(sp.eye(n), t) + sp.kron(t, sp.eye(n))).tocsr()
    a.sort_indices()
    return a.indptr.astype(np.int32), a.indices.astype(np.int32)


def _values(indptr, indices, b, seed):
    rng = np.random.default_rng(seed)
    v = rng.uniform(-1, 1, (indices.size, b, b))
    rows = np.repeat(np.arange(indptr.size - 1), np.diff(indptr))
    v[rows == indices] += 8 * b * np.eye(b)
    return torch.tensor(v.reshape(-1), device="cuda")


@pytest.mark.parametrize("coarse_solve", ["ilu", "dense"])
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [3, 12, 60])
def test_refresh_factors_every_level(n, precision, coarse_solve):
    from aquaflux_gb300.amg import AmgHierarchy

    b = 3
    indptr, indices = _grid(n)
    h = AmgHierarchy(n * n, b, indptr, indices, min_cells=8, precision=precision,
                     coarse_solve=coarse_solve)
    for seed in range(3):  # (the second pass meets factors in place and their graphs)
        fine = _values(indptr, indices, b, seed)
        h.refresh(fine)
        for lv in h.levels if h.dense is None else h.levels[:-1]:
            alone = lv.ilu.clone()
            alone.refactor(lv.values)
            assert torch.equal(lv.ilu.factor_values(), alone.factor_values())
    # the finest level's zero pivot is reported, and the hierarchy can be refreshed again after it
    with pytest.raises(ZeroDivisionError, match="row 0"):
        h.refresh(torch.zeros_like(fine))
    h.refresh(fine)
    assert torch.equal(h.levels[0].ilu.factor_values(), _alone(h.levels[0]))


def _alone(lv):
    alone = lv.ilu.clone()
    alone.refactor(lv.values)
    return alone.factor_values()


# r = rhs - A x is the product and the subtraction, in one pass: bitwise both in turn
@pytest.mark.parametrize("b", [1, 2, 3, 4, 6, 8, 9])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("offset", [0, 1])
def test_residual_is_the_product_and_the_difference(b, dtype, offset):
    from aquaflux_gb300._lib import check, lib, ptr

    indptr, indices = _grid(17)
    n, sfx = 17 * 17, "f32" if dtype == torch.float32 else "f64"
    ip, ix = torch.tensor(indptr, device="cuda"), torch.tensor(indices, device="cuda")
    a = _values(indptr, indices, b, b).to(dtype)
    x = torch.randn(n * b + offset, dtype=dtype, device="cuda")[offset:]
    rhs = torch.randn(n * b + offset, dtype=dtype, device="cuda")[offset:]
    y = torch.empty(n * b, dtype=dtype, device="cuda")
    r = torch.empty_like(y)
    check(getattr(lib(), "fv_bsr_spmv_" + sfx)(n, b, ptr(ip), ptr(ix), ptr(a), ptr(x), ptr(y), 0, 0))
    check(getattr(lib(), "fv_bsr_residual_" + sfx)(n, b, ptr(ip), ptr(ix), ptr(a), ptr(x), ptr(rhs),
                                                   ptr(r), 0))
    torch.cuda.synchronize()
    assert torch.equal(r, rhs - y)
