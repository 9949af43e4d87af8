"""The batched tuner's plan: a forced kernel shape holds for its call alone, and the
calls after it run what they would have run without it."""
import numpy as np
import pytest

import hpc_gb300 as X
from hpc_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("forced", ["0", "5", "7"])  # two CSR shapes, a sliced one
def test_a_forced_shape_does_not_outlive_its_call(gpu_lib, precision, forced, monkeypatch):
    monkeypatch.setenv("XJPCG_BATCH_CLUSTERS", "0")  # the streaming kernels
    batch = W.batched_stencils(count=40, lo=300, hi=3000, seed=8)
    with X.JPCG() as h:
        st, first, _ = h.batch_solve(batch, 20000, 1e-10, precision=precision)
        assert st == X.SUCCESS, h.last_message()
        plan = [getattr(h.info(), f) for f in ("batchThreads", "batchLanes", "batchSliced", "batchSmemRows")]
        monkeypatch.setenv("XJPCG_BATCH_CFG", forced)
        st, _, _ = h.batch_solve(batch, 20000, 1e-10, precision=precision)
        assert st == X.SUCCESS and h.info().batchSliced == (forced == "7")
        monkeypatch.delenv("XJPCG_BATCH_CFG")
        st, again, _ = h.batch_solve(batch, 20000, 1e-10, precision=precision)
        assert st == X.SUCCESS, h.last_message()
        assert plan == [getattr(h.info(), f) for f in ("batchThreads", "batchLanes", "batchSliced", "batchSmemRows")]
        for a, b in zip(first, again):
            assert np.array_equal(a, b)
