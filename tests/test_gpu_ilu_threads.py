"""ILU(0) factors of several host threads at once."""
from __future__ import annotations

import threading

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from tests.test_gpu_amg_refresh import _values

pytestmark = pytest.mark.gpu


def test_one_launch_solves_of_two_sizes_from_two_threads():
    """One block size, so one kernel, with 200 KB of shared memory in one thread and 3 KB in others: no
    launch may see a limit that another has set."""
    from aquaflux_gb300.ilu0 import Ilu0

    errors, threads, done = [], [], threading.Event()

    def work(f, rhs, large):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                r = torch.tensor(rhs, device="cuda")
                want, x = f.solve(r), torch.empty(len(rhs), dtype=torch.float64, device="cuda")
                solves = 0
                while solves < 6000 if large else not done.is_set():
                    f.solve(r, out=x)
                    solves += 1
                stream.synchronize()
                assert torch.equal(x, want)
        except BaseException as e:  # noqa: BLE001 - reported by the test's own thread
            errors.append(e)
        if large:
            done.set()

    for rows in (130, 2, 2, 2, 2):  # 64 columns of cells: level sets of at most 64
        e = [sp.diags([1.0, 1.0, 1.0], [-1, 0, 1], shape=(k, k)) for k in (rows, 64)]
        a = (sp.kron(e[0], sp.eye(64)) + sp.kron(sp.eye(rows), e[1])).tocsr()
        a.sort_indices()
        f = Ilu0.from_csr(a.indptr, a.indices, _values(a.indptr, a.indices, 3, 1), block_size=3)
        rhs = np.random.default_rng(1).uniform(-1, 1, 3 * 64 * rows)
        threads.append(threading.Thread(target=work, args=(f, rhs, rows == 130)))
    torch.cuda.synchronize()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
