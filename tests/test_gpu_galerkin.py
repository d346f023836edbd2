"""Galerkin sums of fp32 blocks (two-float accumulation) against fp64 sums rounded once."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# lists of 0, 1, 2 and many blocks; entries of similar size, spread over more bits than two floats
# hold (summed again in fp64), cancelling, signed zeros, subnormal, infinite and NaN.
@pytest.mark.parametrize("b", [1, 3, 6, 8])
@pytest.mark.parametrize("kind", ["similar", "spread", "cancelling", "special"])
def test_galerkin_sums_are_the_fp64_sums_rounded_once(b, kind):
    from aquaflux_gb300._lib import check, lib, ptr

    rng = np.random.default_rng(b)
    counts = np.array([0, 1, 2, 7, 57, 3, 1, 0, 30] * 20)
    n_fine = 300
    gptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    glist = rng.integers(0, n_fine, gptr[-1]).astype(np.int64)
    fine = rng.uniform(-1, 1, (n_fine, b, b))
    if kind == "spread":
        fine *= 10.0 ** rng.uniform(-30, 30, fine.shape)
    if kind == "cancelling":
        fine[1::2] = -fine[::2] * (1 + 1e-7 * rng.integers(-2, 3, fine[::2].shape))
    if kind == "special":
        pick = rng.integers(0, 40, fine.shape)
        for k, v in enumerate([0.0, -0.0, 1e-42, -3e-45, np.inf, -np.inf, np.nan, 3.3e38]):
            fine[pick == k] = v
    fine = fine.astype(np.float32)
    dev = [torch.tensor(a, device="cuda") for a in (gptr, glist, fine)]
    out = torch.empty(counts.size * b * b, dtype=torch.float32, device="cuda")
    check(lib().fv_galerkin_f32(counts.size, b, ptr(dev[0]), ptr(dev[1]), ptr(dev[2]), 0, ptr(out), 0))
    torch.cuda.synchronize()
    want = np.zeros((counts.size, b, b))
    with np.errstate(all="ignore"):
        for q in range(counts.size):
            for p in range(gptr[q], gptr[q + 1]):  # in list order
                want[q] += fine[glist[p]].astype(np.float64)
        want = want.astype(np.float32).reshape(-1)
    got = out.cpu().numpy()
    ok = np.isnan(want)
    assert np.array_equal(np.isnan(got), ok)
    assert np.array_equal(got[~ok].view(np.int32), want[~ok].view(np.int32))
