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


def _with_a_long_row(extra):
    """7-point rows, one with `extra` more entries; and the dense matrix."""
    rng = np.random.default_rng(4)
    s = W.variable_stencil((11, 11, 12), 1.0, rng)
    a = np.zeros((s.n, s.n))
    a[np.repeat(np.arange(s.n), np.diff(s.rowptr)), s.col] = s.val
    far = rng.choice(np.arange(900, s.n), extra, replace=False)
    a[700, far] = a[far, 700] = -rng.uniform(0.1, 1.0, extra)
    np.fill_diagonal(a, np.abs(a).sum(1) - np.abs(np.diag(a)) + np.diag(a))
    rows, cols = np.nonzero(a)
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=s.n))]).astype(np.int32)
    return W.System(s.n, rowptr, cols.astype(np.int32), a[rows, cols], np.diag(a).copy(), s.b), a


@pytest.mark.parametrize("precision", [0, 1])
def test_uneven_rows_find_the_csr_shapes(gpu_lib, precision, monkeypatch):
    # a row of 300 among rows of 7 holds a slice's other lanes up: the CSR shapes take
    # less than two thirds of the time
    monkeypatch.setenv("XJPCG_BATCH_CLUSTERS", "0")
    hub, a = _with_a_long_row(300)
    with X.JPCG() as h:
        st, xs, res = h.batch_solve([hub] * 400, 20000, 1e-10, precision=precision)
        assert st == X.SUCCESS, h.last_message()
        assert h.info().batchSliced == 0
        for x in xs[:2]:
            assert np.linalg.norm(hub.b - a @ x) <= 1.5e-10 * np.linalg.norm(hub.b)


@pytest.mark.parametrize("name,precision", [("even", 0), ("a_long_row", 1)])
def test_shared_memory_only_where_it_is_faster(gpu_lib, name, precision):
    # as many even systems as fill the GPU twice over, and rows padded to one long row:
    # the streaming kernels take two thirds and a twelfth of the time
    if name == "even":
        batch = [W.variable_stencil((11, 11, 12), 1.0, np.random.default_rng(3))] * 300
    else:
        batch = [_with_a_long_row(100)[0]] * 100
    with X.JPCG() as h:
        st, xs, _ = h.batch_solve(batch, 20000, 1e-10, precision=precision)
        assert st == X.SUCCESS, h.last_message()
        assert h.info().batchSmemRows > 0
        st, ys, _ = h.batch_solve(batch, 20000, 1e-10, precision=precision)
        assert st == X.SUCCESS and h.info().batchSmemRows > 0
        for x, y in zip(xs, ys):
            assert np.array_equal(x, y)
