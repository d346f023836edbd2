"""ILU(0) solves with pivots near the ends of the doubles' range, in every form a solve takes."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from tests.ilu_helpers import oracle_factor_solve

pytestmark = pytest.mark.gpu


# (pivot, its row's next entries, right-hand side of the block): zero unknowns beside a reciprocal out
# of range, cancelling terms each of which overflows once divided, and an entry lost to underflow if
# divided first.  `width` rows a level set: one launch a solve up to 96, a launch a level above.
@pytest.mark.parametrize("width", [1, 96, 97])
@pytest.mark.parametrize("b", [2, 3, 4])
@pytest.mark.parametrize("pivot,entry,rhs", [
    (5e-310, 1.0, (1e-309, 0.0)), (1e-300, 1.0, (1e10, 1e10)), (1e-300, 1e300, (3e-300, 0.0)),
    (1e300, 1e-100, (1e100, 1e200)), (1e-200, -1e200, (1.0, 0.0)), (2.0, 0.0, (6.0, 1.0))])
def test_a_solve_stays_in_range_where_the_operations_in_turn_do(width, b, pivot, entry, rhs):
    from aquaflux_gb300.ilu0 import Ilu0

    layers = 4
    n = width * layers
    i = np.arange(n - width)
    pat = sp.coo_matrix((np.ones(2 * i.size + n), (np.r_[i, i + width, np.arange(n)],
                                                   np.r_[i + width, i, np.arange(n)])), (n, n)).tocsr()
    pat.sort_indices()
    blocks = np.zeros((pat.nnz, b, b))
    block = np.eye(b)
    block[0, 0], block[0, 1] = pivot, entry
    odd = np.arange(n) % 5 == 0  # the other rows are ordinary
    diag = np.repeat(np.arange(n), np.diff(pat.indptr)) == pat.indices
    blocks[diag] = np.where(odd[:, None, None], block, 2.0 * np.eye(b))
    r = np.ones((n, b))
    r[odd] = 0.0
    r[odd, 0], r[odd, 1] = rhs
    a = sp.bsr_matrix((blocks, pat.indices, pat.indptr), shape=(n * b,) * 2)
    full = sp.csr_matrix(np.kron(pat.toarray() != 0, np.ones((b, b))))
    full.sort_indices()
    vals = a.toarray()[np.repeat(np.arange(n * b), np.diff(full.indptr)), full.indices]
    _, _, want, _ = oracle_factor_solve(full.indptr, full.indices, vals, r.reshape(-1))
    assert np.isfinite(want).all()
    f = Ilu0.from_csr(pat.indptr.astype(np.int32), pat.indices.astype(np.int32), blocks.reshape(-1), block_size=b)
    got = f.solve(torch.tensor(r.reshape(-1), device="cuda")).cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=4e-16, atol=0)
