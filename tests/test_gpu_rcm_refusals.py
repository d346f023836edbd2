"""What the renumbering of a malformed graph answers: an error, with nothing written out of range."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3000, 40000])
@pytest.mark.parametrize("first", [0, 1])
def test_rows_that_list_a_node_twice_are_refused(n, first):
    """A path whose rows hold every neighbour twice: each level places its nodes twice, so
    the order overflows, in the seed's component or in one of those after it (node 0 alone)."""
    from aquaflux_gb300._lib import FvError, check, lib, ptr

    rows = [[] for _ in range(n + first)]
    for i in range(first, n + first - 1):
        rows[i] += [i + 1, i + 1]
        rows[i + 1] += [i, i]
    ip = torch.tensor(np.cumsum([0] + [len(r) for r in rows]), dtype=torch.int32, device="cuda")
    ix = torch.tensor([j for r in rows for j in sorted(r)], dtype=torch.int32, device="cuda")
    m = n + first
    perm = torch.full((m,), -7, dtype=torch.int32, device="cuda")
    work = torch.full((3 * m + 65,), -7, dtype=torch.int32, device="cuda")
    seeds = np.arange(m, dtype=np.int64)
    with pytest.raises(FvError, match="inconsistent level size"):
        check(lib().fv_rcm_permutation(m, ptr(ip), ptr(ix), ptr(seeds), ptr(perm), ptr(work), 0))
    torch.cuda.synchronize()
    assert bool((work[3 * m + 1:] == -7).all()) and bool((perm == -7).all())
