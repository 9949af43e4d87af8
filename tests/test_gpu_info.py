"""xJPCG_gbGetInfo on the kernels that ran."""
import pytest

import hpc_gb300 as X
from hpc_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def test_kernels_per_iteration_count_the_hub_copy(gpu_lib, monkeypatch):
    monkeypatch.setenv("XJPCG_SPMV_LANES", "-4")  # length-sorted, unroll 8
    for n, kernels in ((32768, 2), (32769, 3)):  # hubs above 32,768 rows
        s = W.zipf_spd(n, hi=1500, seed=n)
        with X.JPCG() as h:
            r = h.csr_solve(s.n, s.rowptr, s.col, s.val, s.diag, s.b, 2000, 1e-10)
            assert r.status == X.SUCCESS and h.info().spmvLayout == 4
            assert h.info().kernelsPerIter == kernels


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_threads_are_those_of_the_ctas(gpu_lib, precision):
    small, wide = W.poisson7(6), W.poisson7(26)  # the second needs CTAs of the larger kind
    with X.JPCG() as h:
        for batch, threads in (([small] * 3, 128), ([wide], 256 if precision else 448), ([small, wide], 0)):
            st, _, _ = h.batch_solve(batch, 2000, 1e-10, precision=precision)
            assert st == X.SUCCESS and h.info().batchSmemRows == 0
            assert h.info().batchThreads == threads
