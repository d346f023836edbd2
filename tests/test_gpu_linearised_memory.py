"""What a held linearisation of a laminar case keeps on the device: no closure fields."""
from __future__ import annotations

import pytest
import torch

from aquaflux_gb300 import mesh as fm
from aquaflux_gb300 import workloads

pytestmark = pytest.mark.gpu


def test_a_laminar_linearisation_holds_no_closure_fields():
    n = 1000
    bc = {"top": ("moving", (1.0, 0.0)), "bottom": ("wall",), "left": ("wall",), "right": ("wall",)}
    case = workloads.Workload("cavity", fm.structured_grid_2d(n, n), 0.01, 1.0, bc, 0, None).device_case()
    nc, nf, fields, dim = n * n, 2 * n * (n + 1), 3, 2
    s = torch.rand(fields * nc, dtype=torch.float64, device="cuda")
    case.jvp(s, s)  # (what the first pass allocates, and torch for the results)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    case.linearise(s)
    case.jvp_linearised(s, s)
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    # face intermediates and mass-flux estimate; d, gradients and residual
    want = 8 * ((6 + dim + 1) * nf + (1 + fields * dim + fields) * nc)
    assert held <= want + 24 * 2 ** 20, (held, want)  # (allocations come in pieces of 2 MB, torch's of 20)
