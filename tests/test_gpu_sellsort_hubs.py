"""The length-sorted SpMV with hub columns: x at the columns of the longest rows
is read from a compact copy.  Against long-double row sums, on both sides of the
size from which the copy is used."""
import os

import numpy as np
import pytest

import hpc_gb300 as X
from hpc_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FROM = 2 * 16384  # rows above which hubs are used


@pytest.mark.parametrize("n", [FROM, FROM + 1, 50001])
def test_spmv_and_solves_with_hub_columns(gpu_lib, n):
    s = W.zipf_spd(n, hi=1500, seed=n)
    rows, cols, vals = s.coo()
    rng = np.random.default_rng(n)
    env = {"XJPCG_SPMV_LANES": "-4", "XJPCG_GUARD_BYTES": "4096"}
    os.environ.update(env)
    try:
        with X.JPCG() as h:
            r = h.coo_solve(n, rows, cols, vals, s.diag, s.b, 3000, 1e-10)
            assert r.status == X.SUCCESS and h.info().spmvLayout == 4
            v = vals
            for step in range(2):  # the second with new values
                x = rng.uniform(-1.0, 1.0, n)
                y = h.spmv(x)
                prod = v.astype(np.longdouble) * x[cols]
                want = np.add.reduceat(prod, s.rowptr[:-1])
                size = np.add.reduceat(np.abs(prod), s.rowptr[:-1])
                # every product and sum of a row rounds once
                assert np.all(np.abs(y - want) <= (np.diff(s.rowptr) + 1) * 2.0**-53 * size)
                x[cols[s.rowptr[np.argmax(np.diff(s.rowptr))]]] = np.nan
                bad = np.zeros(n, bool)
                bad[rows[np.isnan(x[cols])]] = True
                assert np.array_equal(np.isnan(h.spmv(x)), bad)
                v = 1.5 * v
                r = h.coo_solve(n, None, None, v, 1.5 * s.diag, s.b, 3000, 1e-10, mode=X.MODE_KEEP_NZ_LAYOUT)
                assert r.status == X.SUCCESS
            m = h.mixed_solve(s.b, 1.5 * s.diag, 3000, 1e-10)
            assert m.status == X.SUCCESS
            # converged to 1e-10 each, on a matrix scaled to a condition number of about 1
            assert np.linalg.norm((m.x - r.x) * np.sqrt(s.diag)) <= 1e-8 * np.linalg.norm(r.x * np.sqrt(s.diag))
            assert h.check_guards()[1] == 0
    finally:
        for k in env:
            os.environ.pop(k, None)


def test_without_memory_for_hub_columns_the_solve_goes_on(gpu_lib, monkeypatch):
    # XJPCG_FAULT=hubs: their buffers cannot be had.  The same layout without them
    # sums every row in the same order.
    n = 50001
    s = W.zipf_spd(n, hi=1500, seed=n)
    x = np.random.default_rng(2).uniform(-1.0, 1.0, n)
    monkeypatch.setenv("XJPCG_SPMV_LANES", "-4")
    out = {}
    for fault in ("", "hubs"):
        monkeypatch.setenv("XJPCG_FAULT", fault)
        with X.JPCG() as h:
            r = h.csr_solve(n, s.rowptr, s.col, s.val, s.diag, s.b, 3000, 1e-10)
            assert r.status == X.SUCCESS, r.message
            assert h.info().spmvLayout == 4 and h.info().kernelsPerIter == (2 if fault else 3)
            m = h.mixed_solve(s.b, s.diag, 3000, 1e-10)
            assert m.status == X.SUCCESS, m.message
            out[fault] = h.spmv(x)
    assert np.array_equal(out[""], out["hubs"])


@pytest.mark.parametrize("n", [3001, 50001])
def test_loops_left_to_the_compiler_give_the_same_bits(gpu_lib, n):
    # the last two configurations of the table, after the merge path's
    s = W.zipf_spd(n, hi=1500, seed=n)
    x = np.random.default_rng(3).uniform(-1.0, 1.0, n)
    with X.JPCG() as h:
        h.csr_solve(n, s.rowptr, s.col, s.val, s.diag, s.b, 1, 1e-10)
        shapes = [t[:4] for t in h.spmv_tuning()]
        depths = {u: [c for c, t in enumerate(shapes) if t == (1, 1, u, 32)] for u in (4, 8)}
        assert [c for u in (4, 8) for c in depths[u]][1::2] == [len(shapes) - 2, len(shapes) - 1]
        for u in (4, 8):
            y = []
            for c in depths[u]:
                h.set_spmv_config(c)
                y.append(h.spmv(x))
            assert np.array_equal(y[0], y[1])
