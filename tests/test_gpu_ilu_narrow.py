"""ILU(0) solves with narrow level sets (one launch per solve) against the CPU oracle."""
from __future__ import annotations

import numpy as np
import pytest

from tests.ilu_helpers import oracle_factor_solve

pytestmark = pytest.mark.gpu


def layered(width, layers, b, links, seed):
    """A symmetric block pattern of `layers` level sets of `width` rows, each row coupled to up to `links`
    rows of the layer before; diagonally dominant blocks (condition number below 10)."""
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    n = width * layers
    rows, cols = [np.arange(n)], [np.arange(n)]
    for layer in range(1, layers):
        for i in range(layer * width, (layer + 1) * width):
            j = (layer - 1) * width + np.unique(rng.integers(0, width, links))
            rows += [np.full(j.size, i), j]
            cols += [j, np.full(j.size, i)]
    pat = sp.coo_matrix((np.ones(sum(r.size for r in rows)),
                         (np.concatenate(rows), np.concatenate(cols))), shape=(n, n)).tocsr()
    pat.sort_indices()
    blocks = rng.uniform(-1, 1, (pat.nnz, b, b)) * (0.4 / b)
    for r in range(n):
        q = pat.indptr[r] + int(np.searchsorted(pat.indices[pat.indptr[r]:pat.indptr[r + 1]], r))
        deg = pat.indptr[r + 1] - pat.indptr[r]
        blocks[pat.indptr[r]:pat.indptr[r + 1]] /= deg
        blocks[q] += np.eye(b)
    return pat.indptr.astype(np.int32), pat.indices.astype(np.int32), blocks, rng.standard_normal(n * b)


# a level's rows: one; a partial warp; as many as one launch takes (96 for b <= 4, 48 above) and
# one more (a launch per level).  links: fewer than, as many as and more than a record's blocks (4),
# with remainders of the batches of 2 behind them.  Wider levels: blocks are
# read 4 at a time below 8192 rows (fp32), 2 below 65536, one above.
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("width,layers,b,links", [
    (1, 60, 3, 1), (7, 9, 2, 2), (64, 12, 3, 3), (37, 6, 4, 4), (33, 5, 5, 7), (40, 4, 6, 8), (19, 5, 7, 9),
    (30, 3, 8, 5), (96, 3, 3, 2), (97, 3, 3, 2), (48, 3, 6, 2), (49, 3, 6, 2),
    (8191, 2, 2, 2), (8192, 2, 2, 2), (65535, 2, 2, 1), (65536, 2, 2, 1)])
def test_narrow_level_sets_match_the_oracle(width, layers, b, links, precision):
    """fp64: transposed solve bitwise, forward solve to the rounding of its reordered sums (at most
    links * b + b terms of a well-conditioned row: 100 units in the last place of the largest
    entry); fp32 to 1000 units, its factor being rounded too."""
    import scipy.sparse as sp

    from aquaflux_gb300.ilu0 import Ilu0

    ip, ix, blocks, rhs = layered(width, layers, b, links, 5)
    n = width * layers * b
    a = sp.bsr_matrix((blocks, ix, ip), shape=(n, n)).tocsr()
    a.sort_indices()
    _, _, x, xt = oracle_factor_solve(a.indptr, a.indices, a.data, rhs)
    f = Ilu0.from_csr(ip, ix, blocks.reshape(-1), block_size=b, precision=precision)
    got, got_t = f.solve(rhs).cpu().numpy(), f.solve(rhs, transpose=True).cpu().numpy()
    if precision == 64:
        np.testing.assert_array_equal(got_t, xt)
        np.testing.assert_allclose(got, x, rtol=0, atol=100 * 2.3e-16 * np.abs(x).max())
    else:
        for g, e in ((got, x), (got_t, xt)):
            np.testing.assert_allclose(g, e, rtol=0, atol=1000 * 6e-8 * np.abs(e).max())
    assert np.array_equal(got, f.solve(rhs).cpu().numpy())
    c = f.clone(precision)
    c.refactor(blocks.reshape(-1))
    assert np.array_equal(got, c.solve(rhs).cpu().numpy())


# rows of the factorisation: a warp each, up to 32 columns of a finished row looked up at once, two
# (b <= 4) or four matching blocks updated at once; more than 32 lower blocks, a row too long for
# shared memory (one thread a row), and blocks with zeros (whose quotients are zero).
@pytest.mark.parametrize("n,b,density", [(40, 2, 0.1), (60, 3, 0.3), (50, 4, 1.0), (48, 5, 0.5), (45, 6, 1.0),
                                         (30, 7, 0.4), (24, 8, 1.0), (110, 4, 0.9), (400, 8, 0.02)])
def test_factor_is_bitwise_the_oracle(n, b, density):
    import scipy.sparse as sp

    from aquaflux_gb300.ilu0 import Ilu0

    rng = np.random.default_rng(n + b)
    mask = rng.random((n, n)) < density
    if n == 400:
        mask[0], mask[:, 0] = True, True  # one row of 400 blocks of 512 bytes
    mask = mask | mask.T | np.eye(n, dtype=bool)
    pat = sp.csr_matrix(mask)
    pat.sort_indices()
    blocks = rng.uniform(-1, 1, (pat.nnz, b, b)) * (0.5 / (n * b))
    blocks[rng.random(blocks.shape) < 0.2] = 0.0
    for r in range(n):
        blocks[pat.indptr[r] + int(np.searchsorted(pat.indices[pat.indptr[r]:pat.indptr[r + 1]], r))] += np.eye(b)
    a = sp.bsr_matrix((blocks, pat.indices, pat.indptr), shape=(n * b,) * 2).tocsr()
    rows = np.repeat(np.arange(n), np.diff(pat.indptr))
    full = sp.csr_matrix(np.ones((n * b, n * b)) * np.kron(mask, np.ones((b, b))))
    full.sort_indices()
    dense = a.toarray()
    ip, ix = full.indptr.astype(np.int32), full.indices.astype(np.int32)
    vals = dense[np.repeat(np.arange(n * b), np.diff(ip)), ix]
    _, data, _, _ = oracle_factor_solve(ip, ix, vals, np.ones(n * b))
    f = Ilu0.from_csr(pat.indptr.astype(np.int32), pat.indices.astype(np.int32), blocks.reshape(-1), block_size=b)
    got = f.factor_values().cpu().numpy().reshape(-1, b, b)
    out = np.zeros((n * b, n * b))
    for q, (r, col) in enumerate(zip(rows, pat.indices)):
        out[r * b:(r + 1) * b, col * b:(col + 1) * b] = got[q]
    np.testing.assert_array_equal(out[np.repeat(np.arange(n * b), np.diff(ip)), ix], data)
