"""Solves of several handles from several threads at once.  The fp64 loop as one
kernel holds every SM for a whole solve, so the solves take turns; none may wait
for another until its waits run out, and none may change another's bits."""
import threading

import numpy as np
import pytest

import hpc_gb300 as X
from hpc_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides", [(12, 16), (48, 48), (16, 64, 32)])  # clusters, grids, both
def test_solves_side_by_side(gpu_lib, sides):
    systems = [W.poisson7(side) for side in sides]
    results = [[] for _ in systems]

    def work(k):
        s = systems[k]
        with X.JPCG() as h:
            h.csr_solve(s.n, s.rowptr, s.col, s.val, s.diag, s.b, 0, 1e-10)
            for _ in range(8):
                r = h.csr_solve(s.n, s.rowptr, s.col, s.val, s.diag, s.b, 5000, 1e-10, mode=X.MODE_KEEP_MATRIX)
                results[k].append((r.status, r.message, r.x, h.info().loopUnroll))

    for k in range(len(systems)):  # alone first
        work(k)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(systems))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for got in results:
        assert len(got) == 16
        for status, message, x, unroll in got:
            assert status == X.SUCCESS and unroll == 0, message
            assert np.array_equal(x, got[0][2])
