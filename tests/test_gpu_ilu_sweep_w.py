"""fp32 ILU(0) solves whose level sets take a warp per block row, bitwise the same operations in turn."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F = np.float32


def _pattern(widths, reach, rng):
    """Rows in groups of `widths`; a row couples (both ways) to up to `reach` rows of the groups
    before it, and no two rows of a group to each other: a level set a group."""
    n = sum(widths)
    rows = [{i} for i in range(n)]
    start = 0
    for g, w in enumerate(widths):
        for i in range(start, start + w) if g else ():
            some = rng.choice(start, size=min(reach, start), replace=False)
            for j in [*some, start - 1]:
                rows[i].add(int(j))
                rows[int(j)].add(i)
        start += w
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    return indptr, np.concatenate([sorted(r) for r in rows]).astype(np.int32)


def _solve(indptr, indices, f, r, transpose):
    """The block sweeps in fp32, one operation after the other (lanes of a block side by side)."""
    n, b = indptr.size - 1, f.shape[1]
    x = r.astype(F).reshape(n, b).copy()
    if transpose:
        cols = [[] for _ in range(n)]
        for i in range(n):
            for q in range(indptr[i], indptr[i + 1]):
                cols[indices[q]].append((i, f[q].T))
        row = cols
    else:
        row = [[(indices[q], f[q]) for q in range(indptr[i], indptr[i + 1])] for i in range(n)]
    for i in range(n):
        D = next(m for j, m in row[i] if j == i)
        for j, m in row[i]:
            if j < i:
                for c in range(b):
                    x[i] -= m[:, c] * x[j, c]
        for c in range(b):
            if transpose:
                x[i, c] = x[i, c] / D[c, c]
            x[i, c + 1:] -= D[c + 1:, c] * x[i, c]
    for i in range(n - 1, -1, -1):
        D = next(m for j, m in row[i] if j == i)
        after = [(j, m) for j, m in row[i] if j > i]
        for j, m in reversed(after) if transpose else after:
            for c in range(b - 1, -1, -1) if transpose else range(b):
                x[i] -= m[:, c] * x[j, c]
        for c in range(b - 1, -1, -1):
            if not transpose:
                x[i, c] = x[i, c] / D[c, c]
            x[i, :c] -= D[:c, c] * x[i, c]
    return x.reshape(-1)


# no, few, exactly 32, and more blocks than are held at a time; level sets of 1 row to 150 (wide
# enough that no pattern is solved in one launch)
@pytest.mark.parametrize("b", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("widths,reach", [((150, 149), 2), ((150, 130, 1), 31), ((150, 130, 3), 45)])
def test_warp_per_row_levels_are_the_operations_in_turn(b, widths, reach):
    from aquaflux_gb300.ilu0 import Ilu0

    rng = np.random.default_rng(100 * b + reach)
    indptr, indices = _pattern(widths, reach, rng)
    n = indptr.size - 1
    v = rng.uniform(-1, 1, (indices.size, b, b))
    v[np.repeat(np.arange(n), np.diff(indptr)) == indices] += 40 * b * np.eye(b)
    ilu = Ilu0.from_csr(indptr, indices, torch.tensor(v.reshape(-1), device="cuda"), block_size=b,
                        precision=32)
    f = ilu.factor_values().cpu().numpy().reshape(-1, b, b)
    r = rng.uniform(-1, 1, n * b).astype(F)
    rhs = torch.tensor(r, device="cuda")
    for transpose in (False, True):
        want = _solve(indptr, indices, f, r, transpose)
        got = ilu.solve(rhs, transpose=transpose)
        assert np.array_equal(got.cpu().numpy(), want)
        # recorded into a caller's graph, on another vector and in place
        for in_place in (False, True):
            out = rhs.clone()
            src = out if in_place else rhs
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                ilu.solve(src, transpose=transpose, out=out)
            out.copy_(rhs)
            g.replay()
            assert np.array_equal(out.cpu().numpy(), want)
