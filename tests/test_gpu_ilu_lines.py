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


def _layered(width, layers, links, step=7):
    """`layers` level sets of `width` rows, each row coupled to `links` rows of the one before, `step`
    rows apart (a `step` that divides the width repeats some)."""
    n, off = width * layers, np.arange(links) * step
    i = np.repeat(np.arange(width, n), links)
    j = (i // width - 1) * width + (i % width + np.tile(off, n - width)) % width
    a = sp.coo_matrix((np.ones(2 * i.size + n), (np.r_[i, j, np.arange(n)], np.r_[j, i, np.arange(n)])),
                      (n, n)).tocsr()
    a.sum_duplicates()
    a.sort_indices()
    return a


def _copies(a, k):
    """`k` copies of the pattern that do not couple: level sets k times as wide."""
    c = sp.block_diag([a] * k, format="csr")
    c.sort_indices()
    return c


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


# fp32 b, links: what the line between a warp and 8 lanes a row of the factor sees
@pytest.mark.parametrize("b,links", [(2, 3), (3, 6), (4, 6), (4, 12), (5, 6), (6, 3), (6, 6), (6, 12), (8, 6)])
def test_a_factor_of_narrower_levels_is_not_the_slower_one(b, links):
    """fp32, three level sets from 2,000 to 70,000 rows: no width takes more than 1.2 times what a
    larger one takes."""
    times = []
    for width in (2000, 4000, 6000, 9000, 14000, 22000, 40000, 65000, 70000):
        a = _layered(width, 3, links)
        v = _blocks(a, b, torch.float32)
        f = _factor(a, b, 32, v)
        times.append(_time(lambda: f.refactor(v)))
    for k, t in enumerate(times):
        assert t <= 1.2 * min(times[k:]), (k, times)


@pytest.mark.parametrize("b,links", [(2, 3), (3, 1), (3, 3), (4, 2), (4, 4), (4, 6), (5, 1), (6, 2), (8, 1)])
def test_an_fp64_factor_of_narrower_levels_is_not_the_slower_one(b, links):
    """Twelve level sets of 300 to 3,000 rows: no width takes more than 1.15 times what a larger one does."""
    times = []
    for width in (300, 608, 609, 900, 1023, 1024, 1216, 1217, 1500, 1824, 1825, 2047, 2048, 3000):
        a = _layered(width, 12, links)
        v = _blocks(a, b, torch.float64)
        f = _factor(a, b, 64, v)
        times.append(_time(lambda: f.refactor(v)))
    for k, t in enumerate(times):
        assert t <= 1.15 * min(times[k:]), (k, times)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("b,links", [(2, 3), (3, 6), (4, 16), (5, 1), (6, 3), (6, 12), (7, 6), (8, 3)])
def test_a_factor_is_the_same_at_every_width(b, links, precision):
    """Copies side by side, so that a row's level and with it the kernel is another one: bitwise."""
    dtype = torch.float64 if precision == 64 else torch.float32
    a = _layered(500, 3, links)
    v = _blocks(a, b, dtype, seed=b)
    want = _factor(a, b, precision, v).factor_values()
    for k in (2, 3, 7, 12, 24):  # 1,000 to 12,000 rows a level set
        got = _factor(_copies(a, k), b, precision, v.repeat(k)).factor_values()
        assert torch.equal(got, want.repeat(k)), k


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("b", [2, 4, 6])
def test_a_factor_is_the_same_for_scattered_rows(b, precision):
    """A grid's own order, whose level sets are diagonals of up to 1,200 rows, and its reverse
    Cuthill-McKee-like order by diagonals, whose level sets lie together: bitwise, block by block."""
    dtype = torch.float64 if precision == 64 else torch.float32
    nx, ny, nz = 40, 36, 32
    e = [sp.diags([1.0, 1.0, 1.0], [-1, 0, 1], shape=(k, k)) for k in (nx, ny, nz)]
    i = [sp.eye(k) for k in (nx, ny, nz)]
    a = (sp.kron(sp.kron(e[2], i[1]), i[0]) + sp.kron(sp.kron(i[2], e[1]), i[0]) +
         sp.kron(sp.kron(i[2], i[1]), e[0])).tocsr()
    a.sort_indices()
    q = np.arange(nx * ny * nz)
    p = np.argsort(q // (nx * ny) + q // nx % ny + q % nx, kind="stable")  # ascending on a diagonal
    where = sp.csr_matrix((np.arange(1, a.nnz + 1), a.indices, a.indptr))[p][:, p].tocsr()
    where.sort_indices()
    v = _blocks(a, b, dtype, seed=b)
    block = torch.tensor(where.data - 1, device="cuda")
    f = _factor(a, b, precision, v).factor_values().reshape(-1, b * b)
    g = _factor(where, b, precision, v.reshape(-1, b * b)[block].reshape(-1)).factor_values()
    assert torch.equal(g, f[block].reshape(-1))


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("b,links", [(2, 1), (2, 8), (3, 2), (3, 4), (3, 20), (4, 1), (4, 2), (4, 8), (4, 20)])
def test_a_solve_of_narrow_levels_is_not_the_slower_one(b, links, transpose):
    """fp64, 60 level sets of 16 to 97 rows, in one launch or one a level: no width takes more than 1.15
    times what a larger one takes."""
    times = []
    for width in (16, 32, 40, 48, 56, 64, 80, 96, 97):
        a = _layered(width, 60, links, 1)
        f = _factor(a, b, 64, _blocks(a, b, torch.float64))
        r = torch.rand(width * 60 * b, device="cuda", dtype=torch.float64)
        x = torch.empty_like(r)
        times.append(_time(lambda: f.solve(r, transpose=transpose, out=x)))
    for k, t in enumerate(times):
        assert t <= 1.15 * min(times[k:]), (k, times)


@pytest.mark.parametrize("b,links", [(2, 1), (2, 8), (3, 2), (3, 8), (4, 2), (4, 20)])
def test_a_narrow_solve_is_the_same_at_every_width(b, links):
    """Copies side by side, fp64: level sets of 20 to 100 rows, in one launch or one a level.  The
    transposed solve bitwise; the forward one to the rounding of its reordered sums (at most
    links * b + b terms a row of well-conditioned blocks: 100 units in the last place)."""
    a = _layered(20, 30, links, 1)
    v = _blocks(a, b, torch.float64, seed=b)
    r = torch.rand(600 * b, device="cuda", dtype=torch.float64) - 0.5
    f = _factor(a, b, 64, v)
    x, xt = f.solve(r), f.solve(r, transpose=True)
    for k in (2, 3, 4, 5):
        g = _factor(_copies(a, k), b, 64, v.repeat(k))
        assert torch.equal(g.solve(r.repeat(k), transpose=True), xt.repeat(k)), k
        d = float((g.solve(r.repeat(k)) - x.repeat(k)).abs().max())
        assert d <= 100 * 2.3e-16 * float(x.abs().max()), (k, d)


# rows of 14 blocks beside the diagonal one: their reading is most of a level's time
@pytest.mark.parametrize("b,precision", [(2, 64), (3, 64), (4, 64), (5, 64), (2, 32), (3, 32), (4, 32), (5, 32), (7, 32)])
@pytest.mark.parametrize("transpose", [False, True])
def test_a_solve_of_narrower_levels_is_not_the_slower_one(b, precision, transpose):
    """Six level sets of 511 to 12,000 rows: no width takes more than 1.12 times what a larger one does."""
    dtype = torch.float64 if precision == 64 else torch.float32
    times = []
    for width in (511, 512, 1024, 1025, 2047, 2049, 3073, 5000, 8191, 8192, 12000):
        a = _layered(width, 6, 14)
        f = _factor(a, b, precision, _blocks(a, b, dtype))
        r = torch.rand(a.shape[0] * b, device="cuda", dtype=dtype)
        x = torch.empty_like(r)
        times.append(_time(lambda: f.solve(r, transpose=transpose, out=x), 25))
    for k, t in enumerate(times):
        assert t <= 1.12 * min(times[k:]), (k, times)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("b,links", [(2, 3), (3, 3), (3, 14), (4, 16), (5, 3), (5, 9), (6, 3), (6, 12), (7, 6), (8, 10)])
def test_a_solve_is_the_same_at_every_width(b, links, precision):
    """Copies side by side and blocks said to come from memory or not, so that a row's level takes every
    form of reading (from 100 rows, more than one launch a solve takes, to 72,000): bitwise."""
    dtype = torch.float64 if precision == 64 else torch.float32
    a = _layered(100, 3, links)
    v = _blocks(a, b, dtype, seed=b)
    r = torch.rand(300 * b, device="cuda", dtype=dtype) - 0.5
    f = _factor(a, b, precision, v)
    want = [f.solve(r, transpose=t) for t in (False, True)]
    for k in (1, 5, 6, 11, 20, 31, 50, 90, 200, 400, 720):
        if precision == 64 and k > 20:
            break
        g = _factor(_copies(a, k), b, precision, v.repeat(k))
        for traffic in (0, 120_000_000, 10**9):
            g.set_traffic(traffic)
            for t in (False, True):
                assert torch.equal(g.solve(r.repeat(k), transpose=t), want[t].repeat(k)), (k, traffic, t)


# the widths at which fp64 levels change their reading, rows of 11 and 22 blocks on a side (read two at a
# time, with a remainder, or as the compiler unrolls them)
@pytest.mark.parametrize("b,links", [(2, 11), (3, 11), (4, 11), (3, 22)])
@pytest.mark.parametrize("width", [511, 512, 1024, 1025])
def test_long_rows_on_both_sides_of_a_reading_match_the_oracle(width, b, links):
    """The factor and the transposed solve bitwise; the forward solve to the rounding of its reordered
    sums (at most links * b + b terms a row of well-conditioned blocks: 100 units in the last place)."""
    from tests.ilu_helpers import oracle_factor_solve

    a = _layered(width, 3, links)
    v = _blocks(a, b, torch.float64, seed=width)
    full = sp.bsr_matrix((v.cpu().numpy().reshape(-1, b, b), a.indices, a.indptr)).tocsr()
    full.sort_indices()
    rhs = np.random.default_rng(width).uniform(-1, 1, a.shape[0] * b)
    _, data, x, xt = oracle_factor_solve(full.indptr, full.indices, full.data, rhs)
    f = _factor(a, b, 64, v)
    got = sp.bsr_matrix((f.factor_values().cpu().numpy().reshape(-1, b, b), a.indices, a.indptr)).tocsr()
    got.sort_indices()
    assert np.array_equal(got.data, data)
    r = torch.tensor(rhs, device="cuda")
    for traffic in (0, 10**9):
        f.set_traffic(traffic)
        assert np.array_equal(f.solve(r, transpose=True).cpu().numpy(), xt)
        np.testing.assert_allclose(f.solve(r).cpu().numpy(), x, rtol=0, atol=100 * 2.3e-16 * np.abs(x).max())
