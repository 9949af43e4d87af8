"""The fp64 loop as one kernel (over the grid, or in one cluster for small
systems) against the host-driven loop of the same layout.  Rows are summed in
the same order in both; only the order of the dot products differs, so a few
iterations agree to rounding and converged solves to the solver's bar.  Inside
the kernel neither the layout nor what is kept in shared memory may change a
bit."""
import os

import numpy as np
import pytest

import hpc_gb300 as X
from hpc_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# (extents, 7-point stencil, kernel: "cluster", "grid" or "graph")
SYSTEMS = {
    "one_row": ((1, 1, 1), True, "cluster"),
    "three_rows": ((1, 1, 3), False, "cluster"),
    "one_slice": ((2, 4, 4), False, "cluster"),
    "slice_and_a_row": ((1, 3, 11), True, "cluster"),
    "uneven_rows": ((7, 8, 9), False, "cluster"),
    "largest_cluster": ((24, 24, 25), True, "cluster"),
    "smallest_grid": ((25, 25, 25), True, "grid"),
    "a_slice_per_sm_and_one": ((17, 13, 23), False, "cluster"),
    "wide_plane": ((3, 190, 191), True, "grid"),  # columns beyond int16 offsets
    "matrix_just_on_chip": ((47, 48, 49), False, "grid"),
    "matrix_partly_on_chip": ((79, 80, 81), True, "grid"),
    "steps_of_9": ((2, 310, 311), False, "grid"),  # 18 entries a row, no int16 offsets
    "steps_of_7_and_5": ((2, 2, 7001), False, "grid"),
    "empty_slices": ((20, 21, 23), False, "grid"),
    "J_just_on_chip": ((94, 95, 95), True, "grid"),
    "J_not_on_chip": ((96, 97, 97), True, "grid"),
    "vectors_too_large": ((103, 103, 104), True, "graph"),
}


def _system(shape, seven):
    rng = np.random.default_rng(sum(shape) + seven)
    offs = [d for d in W._grid_dirs(3) if not seven or sum(abs(o) for o in d) == 1]
    pair = {}
    for d in [d for d in offs if d > (0, 0, 0)]:
        src, _ = W._slices(shape, d)
        pair[d] = rng.lognormal(0.0, 1.0, tuple(max(0, s.stop - s.start) for s in src))
    s = W.stencil_system(shape, offs, pair, rng.lognormal(0.0, 1.0, shape))
    s.b = rng.uniform(-1.0, 1.0, s.n)
    return s


def _solves(s, env, calls):
    env = dict(env, XJPCG_GUARD_BYTES="4096")
    os.environ.update(env)
    out = []
    try:
        with X.JPCG() as h:
            rows, cols, vals = s.coo()
            h.coo_solve(s.n, rows, cols, vals, s.diag, s.b, 0, 1e-10)
            for max_iter, tol in calls:
                r = h.coo_solve(s.n, None, None, None, s.diag, s.b, max_iter, tol, mode=X.MODE_KEEP_MATRIX)
                out.append((r, h.records(), h.info()))
            assert h.check_guards()[1] == 0
    finally:
        for k in env:
            os.environ.pop(k, None)
    return out


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_loop_kernel_matches_the_host_loop(gpu_lib, name):
    shape, seven, form = SYSTEMS[name]
    s = _system(shape, seven)
    if name == "empty_slices":  # rows without stored entries, where b is 0
        s.n, s.diag, s.b = s.n + 100, np.append(s.diag, np.ones(100)), np.append(s.b, np.zeros(100))
        s.rowptr = np.append(s.rowptr, np.full(100, s.rowptr[-1]))
    few = min(4, s.n)  # short of convergence, where the steps stay well conditioned
    calls = [(few - 1, 1e-30), (3000, 1e-10), (3000, 1e-10)]
    host = _solves(s, {"XJPCG_SPMV_LANES": "-1", "XJPCG_HOST_LOOP": "1"}, calls)
    default = _solves(s, {}, calls)
    runs = [default]
    for lanes in ("-1", "-5") if name in ("wide_plane", "steps_of_9") else ("-1", "-3", "-5"):
        runs.append(_solves(s, {"XJPCG_SPMV_LANES": lanes, "XJPCG_LOOP_KERNEL": "1"}, calls))
    for run in runs:
        (ra, reca, ia), (rb, _, _), (rc, _, _) = run
        assert (ia.loopUnroll == 0) == (form != "graph")
        # n rounding errors in each sum, a few steps: 1e-11 is far above
        assert ra.iters == host[0][0].iters and ia.itersRun == few
        assert np.linalg.norm(ra.x - host[0][0].x) <= 1e-11 * np.linalg.norm(host[0][0].x)
        for f in ("id", "iter", "vecSize", "maxIter"):
            assert np.array_equal(reca[f], host[0][1][f]), f
        if s.n > 3:
            for f in ("tols", "res", "rz", "alpha", "beta"):
                assert np.allclose(reca[f], host[0][1][f], rtol=1e-9, atol=0), f
        # converged: the solver's bar
        h = host[1][0]
        assert rb.status == h.status == X.SUCCESS, rb.message
        assert abs(rb.iters - h.iters) <= max(1, 0.01 * h.iters)
        assert np.linalg.norm(rb.x - h.x) <= 1e-8 * np.linalg.norm(h.x)
        # the same bits again, and whatever the layout
        assert rc.iters == rb.iters and np.array_equal(rb.x, rc.x)
        if form != "graph":
            assert rb.iters == default[1][0].iters and np.array_equal(rb.x, default[1][0].x)


@pytest.mark.parametrize("shape", [(10, 11, 12), (30, 31, 32)])  # cluster, grid
def test_loop_kernel_limits_and_breakdown(gpu_lib, shape):
    s = _system(shape, True)
    for limit in (0, 1, 7):
        (a, _, ia), = _solves(s, {}, [(limit, 1e-10)])
        (b, _, ib), = _solves(s, {"XJPCG_HOST_LOOP": "1"}, [(limit, 1e-10)])
        assert a.status == b.status == X.EXECUTION_FAILED
        assert a.iters == b.iters == limit and ia.itersRun == ib.itersRun == limit + 1
        assert np.linalg.norm(a.x - b.x) <= 1e-11 * np.linalg.norm(b.x)
    with X.JPCG() as h:
        rows, cols, vals = s.coo()
        good = h.coo_solve(s.n, rows, cols, vals, s.diag, s.b, 2000, 1e-10)
        for bad in (np.nan, np.inf, 0.0):
            b = np.zeros(s.n) if bad == 0.0 else s.b.copy()
            b[17] = bad
            r = h.coo_solve(s.n, None, None, None, s.diag, b, 50, 1e-10, mode=X.MODE_KEEP_MATRIX)
            assert r.status == X.EXECUTION_FAILED and h.info().itersRun == 1
        again = h.coo_solve(s.n, None, None, None, s.diag, s.b, 2000, 1e-10, mode=X.MODE_KEEP_MATRIX)
        assert again.status == X.SUCCESS and np.array_equal(good.x, again.x)
