"""The two halves of an ILU(0) factorisation: what is refused while one is started."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.test_gpu_amg_refresh import _grid, _values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
def test_a_started_factor_is_not_read_or_written_before_its_finish(precision):
    from aquaflux_gb300._lib import FvError
    from aquaflux_gb300.ilu0 import Ilu0

    ip, ix = _grid(20)
    b = 3
    f = Ilu0.from_csr(ip, ix, _values(ip, ix, b, 1), block_size=b, precision=precision)
    new = _values(ip, ix, b, 2)
    want = Ilu0.from_csr(ip, ix, new, block_size=b, precision=precision)
    r = torch.tensor(np.ones(400 * b), dtype=want.factor_values().dtype, device="cuda")
    with pytest.raises(FvError, match="no factorisation was started"):
        f.finish_factor()
    held = f.start_factor(new)
    for call in (lambda: f.solve(r), lambda: f.solve(r, transpose=True), f.factor_values,
                 lambda: f.refactor(new), lambda: f.start_factor(new)):
        with pytest.raises(FvError, match="fv_ilu0_factor_finish has to follow"):
            call()
    copy = f.clone(precision)  # the pattern only
    f.finish_factor()
    del held
    assert torch.equal(f.factor_values(), want.factor_values())
    assert torch.equal(f.solve(r), want.solve(r))
    assert torch.equal(f.solve(r, transpose=True), want.solve(r, transpose=True))
    with pytest.raises(FvError, match="no factorisation was started"):
        f.finish_factor()
    copy.start_factor(new)
    del copy  # destroyed with its factorisation started
    torch.cuda.synchronize()
