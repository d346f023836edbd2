"""ILU(0) and block products on both sides of what chooses their kernel: one side may not be much
slower than the other, and both give the same results."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


def _time(f, n=15):
    """The least of n runs, in seconds."""
    f()
    best = np.inf
    for _ in range(n):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        f()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e-3)
    return best


def _blocks(a, b, dtype, seed=0):
    """Diagonally dominant blocks on the pattern of ``a``."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.rand(a.nnz, b, b, device="cuda", generator=g, dtype=torch.float64) - 0.5
    d = np.flatnonzero(np.repeat(np.arange(a.shape[0]), np.diff(a.indptr)) == a.indices)
    v[torch.tensor(d, device="cuda")] += b * float(np.diff(a.indptr).max()) * torch.eye(b, device="cuda")
    return v.reshape(-1).to(dtype)


def _factor(a, b, precision, v):
    from aquaflux_gb300.ilu0 import Ilu0

    return Ilu0.from_csr(a.indptr.astype(np.int32), a.indices.astype(np.int32), v, block_size=b,
                         precision=precision)


@pytest.mark.parametrize("b,precision", [(6, 64), (8, 64), (8, 32)])
def test_one_long_row_costs_the_factor_its_own_level_only(b, precision):
    """A 96 x 96 grid, and the same with the first cell coupled to 400 others (a row of more blocks than
    fit a warp's share of shared memory): at most twice the time, for 1 % more blocks."""
    dtype = torch.float64 if precision == 64 else torch.float32
    e = sp.diags([1.0, 1.0, 1.0], [-1, 0, 1], shape=(96, 96))
    grid = (sp.kron(e, sp.eye(96)) + sp.kron(sp.eye(96), e)).tolil()
    times = []
    for more in (0, 400):
        grid[0, 1:1 + 20 * more:20] = 1.0
        a = grid.tocsr()
        a.sort_indices()
        v = _blocks(a, b, dtype)
        f = _factor(a, b, precision, v)
        times.append(_time(lambda: f.refactor(v)))
    assert times[1] <= 2.0 * times[0], times
