"""Block products and defects by every kernel that computes them, on both sides of what chooses it."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F = np.float32


def _rows(n, counts, rng):
    """`n` rows of the given numbers of blocks, at ascending random columns."""
    counts = np.resize(counts, n)
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    indices = np.concatenate([np.sort(rng.choice(n, c, replace=False)) for c in counts]).astype(np.int32)
    return indptr, indices


# rows of fewer, exactly and more blocks than are held at a time (32), and of none; few rows take a warp
# a row and many a thread a scalar row; `known`: the pattern's counts passed, its size, or neither
@pytest.mark.parametrize("b", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("n,counts", [(70, (33, 0, 1, 65)), (301, (32, 7)), (511, (5,)), (512, (5, 3)), (4600, (9, 7)),
                                      (6143, (7,)), (6144, (3, 40))])
def test_products_are_the_operations_in_turn(b, n, counts):
    from aquaflux_gb300._lib import check, lib, ptr
    from aquaflux_gb300.sparse import bsr_spmv

    rng = np.random.default_rng(n + b)
    indptr, indices = _rows(n, counts, rng)
    a = rng.uniform(-1, 1, (indices.size, b, b)).astype(F)
    x, rhs = rng.uniform(-1, 1, n * b).astype(F), rng.uniform(-1, 1, n * b).astype(F)
    want, xb, nq = np.zeros((n, b), F), x.reshape(n, b), np.diff(indptr)
    for k in range(nq.max()):  # block k of the rows that have it, a product and an addition in turn
        i = np.flatnonzero(nq > k)
        q = indptr[i] + k
        for c in range(b):
            want[i] += a[q][:, :, c] * xb[indices[q], c][:, None]
    want = want.reshape(-1)
    d = [torch.tensor(v, device="cuda") for v in (indptr, indices, a.reshape(-1), x, rhs)]
    ip, ix, av, xv, rv = map(ptr, d)
    y = torch.empty(n * b, device="cuda")
    calls = [lambda r: lib().fv_bsr_product_f32(n, b, indices.size, int(nq.max()), 0, ip, ix, av, xv, r, ptr(y), 0),
             lambda r: lib().fv_bsr_product_f32(n, b, indices.size, int(nq.max()), 10**9, ip, ix, av, xv, r, ptr(y), 0),
             lambda r: lib().fv_bsr_product_f32(n, b, indices.size, 0, 0, ip, ix, av, xv, r, ptr(y), 0),
             lambda r: (lib().fv_bsr_residual_f32(n, b, ip, ix, av, xv, r, ptr(y), 0) if r else
                        lib().fv_bsr_spmv_f32(n, b, ip, ix, av, xv, ptr(y), 0, 0))]
    for call in calls:
        check(call(None))
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy(), want)
        check(call(rv))
        torch.cuda.synchronize()
        assert np.array_equal(y.cpu().numpy(), rhs - want)
    assert np.array_equal(bsr_spmv(d[0], d[1], d[2], b, d[3]).cpu().numpy(), want)


@pytest.mark.parametrize("b,k", [(3, 5), (3, 7), (4, 5), (4, 7), (5, 5), (6, 5), (6, 7), (6, 14), (6, 27), (7, 7), (8, 7)])
def test_a_product_of_fewer_rows_is_not_the_slower_one(b, k):
    """fp32, 250 to 6,500 rows of k blocks: no size takes more than 1.15 times what a larger one does."""
    from aquaflux_gb300.sparse import bsr_spmv

    times = []
    for n in (250, 511, 600, 1000, 1600, 2300, 3000, 3700, 4700, 6143, 6144, 6500):
        ix = np.sort((np.arange(n)[:, None] + np.r_[np.arange(-2, 3), 16 * np.arange(1, k)][:k]) % n, axis=1)
        ip = torch.arange(0, n * k + 1, k, dtype=torch.int32, device="cuda")
        ix = torch.tensor(ix.reshape(-1), dtype=torch.int32, device="cuda")
        a, x = torch.rand(n * k * b * b, device="cuda"), torch.rand(n * b, device="cuda")
        y = torch.empty_like(x)
        bsr_spmv(ip, ix, a, b, x, out=y)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(40):
                bsr_spmv(ip, ix, a, b, x, out=y)
        best = np.inf
        for _ in range(12):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda.synchronize()
            e[0].record()
            g.replay()
            e[1].record()
            e[1].synchronize()
            best = min(best, e[0].elapsed_time(e[1]) * 25.0)
        times.append(best)
    for i, t in enumerate(times):
        assert t <= 1.15 * min(times[i:]), (i, times)
