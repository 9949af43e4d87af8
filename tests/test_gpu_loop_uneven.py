"""The fp64 loop as one kernel on uneven rows and scattered columns: where it is
taken, where the graph loop is the faster one, and that both agree with the
host-driven loop."""
import os

import numpy as np
import pytest

import hpc_gb300 as X
from hpc_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _spd(n, i, j, w):
    """Symmetric, diagonally dominant, from entries (i, j) in any order."""
    lo, hi = np.minimum(i, j), np.maximum(i, j)
    key, at = np.unique(lo * n + hi, return_index=True)
    keep = key // n != key % n
    lo, hi, w = key[keep] // n, key[keep] % n, w[at[keep]]
    diag = 1.02 * (np.bincount(lo, np.abs(w), n) + np.bincount(hi, np.abs(w), n)) + 0.5
    r, c = np.concatenate([lo, hi, np.arange(n)]), np.concatenate([hi, lo, np.arange(n)])
    v = np.concatenate([w, w, diag])
    order = np.argsort(r * n + c, kind="stable")
    rowptr = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(r, minlength=n), out=rowptr[1:])
    b = np.random.default_rng(n).uniform(-1.0, 1.0, n)
    return W.System(n, rowptr, c[order].astype(np.int32), v[order], diag, b)


def _random(n, lo, hi, seed, order=None):
    """Rows of about lo .. hi entries in random columns; ascending where asked."""
    rng = np.random.default_rng(seed)
    length = rng.integers(lo, hi + 1, n) // 2
    i = np.repeat(np.arange(n), np.sort(length) if order else length)
    return _spd(n, i, rng.integers(0, n, i.size), rng.normal(size=i.size))


def _grid(side, seven=True, long_row=0, shuffled=False):
    n, rng = side**3, np.random.default_rng(side)
    at = np.arange(n).reshape(side, side, side)
    i, j = [], []
    for d in W._grid_dirs(3):
        if d > (0, 0, 0) and (not seven or sum(abs(o) for o in d) == 1):
            src, dst = W._slices(at.shape, d)
            i.append(at[src].ravel())
            j.append(at[dst].ravel())
    i, j = np.concatenate(i), np.concatenate(j)
    if shuffled:
        place = rng.permutation(n)
        i, j = place[i], place[j]
    if long_row:
        i = np.concatenate([i, np.full(long_row, n // 2)])
        j = np.concatenate([j, rng.choice(n, long_row, replace=False)])
    return _spd(n, i, j, rng.normal(size=i.size))


SYSTEMS = {
    # rows long or uneven enough for every layout to be timed: a lane per row is too slow
    "rows_of_400_to_700": (lambda: _random(2000, 400, 900, 1), "graph"),
    "a_row_of_600": (lambda: _grid(37, long_row=600), "graph"),
    "a_row_of_300": (lambda: _grid(20, long_row=300), "graph"),
    # near enough to even
    "a_row_of_120": (lambda: _grid(16, long_row=120), "one kernel"),
    "ascending_rows": (lambda: _random(20000, 4, 20, 2, order=True), "one kernel"),
    # scattered columns: over the grid, or in a cluster when they are few
    "scattered": (lambda: _random(4000, 32, 32, 3), "one kernel"),
    "scattered_few": (lambda: _random(1000, 32, 32, 4), "one kernel"),
    "shuffled_27_point": (lambda: _grid(16, seven=False, shuffled=True), "one kernel"),
    # two dense slices: one CTA of a cluster could not hold them
    "two_dense_slices": (lambda: _spd(1000, np.repeat(np.arange(64), 936), np.tile(np.arange(64, 1000), 64),
                                      np.random.default_rng(5).normal(size=64 * 936)), "one kernel"),
}


def _solves(s, calls, **env):
    env["XJPCG_GUARD_BYTES"] = "4096"
    os.environ.update(env)
    try:
        with X.JPCG() as h:
            h.csr_solve(s.n, s.rowptr, s.col, s.val, s.diag, s.b, 0, 1e-10)
            out = []
            for max_iter, tol in calls:
                r = h.csr_solve(s.n, s.rowptr, s.col, s.val, s.diag, s.b, max_iter, tol, mode=X.MODE_KEEP_MATRIX)
                out.append((r, h.info()))
            assert h.check_guards()[1] == 0
            return out
    finally:
        for k in env:
            os.environ.pop(k, None)


@pytest.mark.parametrize("name", list(SYSTEMS))
def test_uneven_rows_and_scattered_columns(gpu_lib, name):
    make, route = SYSTEMS[name]
    s = make()
    calls = [(3, 1e-30), (3000, 1e-10), (3000, 1e-10)]
    host = _solves(s, calls, XJPCG_HOST_LOOP="1")
    got = _solves(s, calls)
    assert (got[0][1].loopUnroll == 0) == (route == "one kernel")
    # a few steps: rounding of sums of a few hundred products, 1e-11 is far above
    assert np.linalg.norm(got[0][0].x - host[0][0].x) <= 1e-11 * np.linalg.norm(host[0][0].x)
    a, b = got[1][0], host[1][0]
    assert a.status == b.status == X.SUCCESS, a.message
    assert abs(a.iters - b.iters) <= max(1, 0.01 * b.iters)
    assert np.linalg.norm(a.x - b.x) <= 1e-8 * np.linalg.norm(b.x)
    assert np.array_equal(a.x, got[2][0].x)
