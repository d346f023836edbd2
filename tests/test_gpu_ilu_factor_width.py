"""fp64 block factors on both sides of the level widths that choose their kernel, against the scalar one."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu


# level sets of `width` rows, each coupled to three rows of the one before: bitwise the scalar
# elimination of the expanded matrix, which takes one thread a row at every width; then a solve of
# the same levels, to the rounding of some 20 terms a row through three levels
@pytest.mark.parametrize("b", [2, 4, 5, 6])
@pytest.mark.parametrize("width", [152, 153, 511, 512, 1023, 1024, 2047, 2048])
def test_block_factor_is_the_scalar_one(b, width):
    from aquaflux_gb300.ilu0 import Ilu0

    rng = np.random.default_rng(width + b)
    n = 3 * width
    rows, cols = [np.arange(n)], [np.arange(n)]
    for g in (1, 2):
        i = np.repeat(np.arange(g * width, (g + 1) * width), 3)
        j = (i - width) // width * width + (i % width + np.tile([0, 1, 7], width)) % width
        rows += [i, j]
        cols += [j, i]
    a = sp.csr_matrix((np.ones(sum(r.size for r in rows)), (np.concatenate(rows), np.concatenate(cols))), (n, n))
    a.sort_indices()
    v = rng.uniform(-1, 1, (a.nnz, b, b))
    v[np.repeat(np.arange(n), np.diff(a.indptr)) == a.indices] += 8 * b * np.eye(b)
    block = Ilu0.from_csr(a.indptr, a.indices, torch.tensor(v.reshape(-1), device="cuda"), block_size=b)
    full = sp.bsr_matrix((v, a.indices, a.indptr)).tocsr()
    full.sort_indices()
    scalar = Ilu0(full)
    want = sp.csr_matrix((scalar.factor_values().cpu().numpy(), full.indices, full.indptr)).tobsr((b, b))
    want.sort_indices()
    assert np.array_equal(block.factor_values().cpu().numpy(), want.data.reshape(-1))
    r = torch.tensor(rng.uniform(-1, 1, n * b), device="cuda")
    for transpose in (False, True):
        x, y = block.solve(r, transpose=transpose), scalar.solve(r, transpose=transpose)
        assert float((x - y).abs().max()) <= 1e-13 * float(y.abs().max())
