"""Batches solved from shared memory (one CTA or cluster per system) and the
teams of the streaming kernels, against the oracle."""
import numpy as np
import pytest

import hpc_gb300 as X
import oracle
from hpc_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _stencil(shape, seed):
    return W.variable_stencil(shape, 1.0, np.random.default_rng(seed))


def _scattered(n, reach, per_row, seed):
    """Random symmetric SPD matrix: rows of uneven length, columns in no pattern."""
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), per_row)
    j = (i + rng.integers(-reach, reach + 1, i.size)) % n
    lo, hi = np.minimum(i, j), np.maximum(i, j)
    key = np.unique((lo * n + hi)[lo != hi])
    lo, hi = key // n, key % n
    w = rng.normal(size=key.size)
    diag = 1.05 * (np.bincount(lo, np.abs(w), n) + np.bincount(hi, np.abs(w), n)) + 0.5
    r, c = np.concatenate([lo, hi, np.arange(n)]), np.concatenate([hi, lo, np.arange(n)])
    v = np.concatenate([w, w, diag])
    order = np.argsort(r * n + c, kind="stable")
    rowptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=rowptr[1:])
    return W.System(n, rowptr.astype(np.int32), c[order].astype(np.int32), v[order], diag, rng.uniform(-1, 1, n))


BATCHES = {
    # rows at the edges of a slice, of a small CTA (512) and of two of them
    "edges": lambda: [_stencil((1, m), m) for m in (2, 31, 32, 33, 64)] + [_stencil((32, 16), 1),
                      _stencil((27, 19), 2), _stencil((32, 32), 3), _stencil((25, 41), 4), _stencil((8, 8, 8), 5)],
    # clusters of small CTAs, their largest (8,192 rows) and the wide CTAs beyond
    "clusters": lambda: [_stencil((46, 47), 6), _stencil((16, 16, 16), 7), _stencil((64, 128), 8),
                         _stencil((67, 123), 9), _stencil((25, 26, 27), 10)],
    # no shared offsets, columns far outside the CTA, more than eight per row
    # (an entry count too large for shared memory takes the other kernels)
    "scattered": lambda: [_scattered(700, 700, 3, 11), _scattered(2500, 2500, 6, 12), _scattered(1300, 40, 9, 13)],
    "one_row": lambda: [_scattered(1, 0, 1, 14), _scattered(2, 1, 2, 15)],
}


def _check(batch, xs, res, precision):
    for s, x, r in zip(batch, xs, res):
        ref = oracle.jpcg(s.rowptr, s.col, s.val, s.diag, s.b, 20000, 1e-10)
        assert r["status"] == 0
        assert oracle.true_relres(s.rowptr, s.col, s.val, s.b, x) <= 1.5e-10
        assert np.linalg.norm(x - ref["x"]) <= 1e-8 * np.linalg.norm(ref["x"])
        if precision == 0:
            assert abs(int(r["iters"]) - ref["iters"]) <= max(1, int(0.01 * ref["iters"]))
        else:
            assert int(r["iters"]) <= 1.25 * ref["iters"] + 5 and r["outer"] >= 1


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", list(BATCHES))
def test_batched_from_shared_memory(gpu_lib, name, precision, monkeypatch):
    monkeypatch.setenv("XJPCG_GUARD_BYTES", "4096")
    batch = BATCHES[name]()
    with X.JPCG() as h:
        # the fewest CTAs (beside enough systems to fill the GPU), then the most
        many = batch * max(1, 400 // len(batch)) if name in ("edges", "one_row") else batch
        for sub in (many, batch):
            st, xs, res = h.batch_solve(sub, 20000, 1e-10, precision=precision)
            assert st == X.SUCCESS, h.last_message()
            assert h.info().batchSmemRows == 0  # solved from shared memory
            _check(batch, xs, res, precision)
            for k, x in enumerate(xs):  # copies of a system agree bit for bit
                assert np.array_equal(x, xs[k % len(batch)])
        # a cap of 5 iterations is reported as xJPCG does
        if name != "one_row":  # (those are solved exactly in two)
            st, _, res = h.batch_solve(batch[-1:], 5, 1e-30, precision=precision)
            assert st == X.EXECUTION_FAILED and int(res[0]["itersRun"]) <= 6
        assert h.check_guards()[1] == 0


@pytest.mark.parametrize("precision", [0, 1])
def test_batched_teams(gpu_lib, precision, monkeypatch):
    # long systems on teams of CTAs beside short ones
    monkeypatch.setenv("XJPCG_BATCH_CLUSTERS", "0")
    monkeypatch.setenv("XJPCG_BATCH_TEAMS", "1")
    monkeypatch.setenv("XJPCG_GUARD_BYTES", "4096")
    batch = [_stencil((20, 21), k) for k in range(6)] + [_stencil((47, 48), 20), _stencil((70, 71), 21),
             _stencil((93, 99), 22), _stencil((21, 22, 23), 23), _scattered(5000, 5000, 5, 24)]
    with X.JPCG() as h:
        st, xs, res = h.batch_solve(batch, 20000, 1e-10, precision=precision)
        assert st == X.SUCCESS, h.last_message()
        assert h.info().batchGrid <= 8 * 8  # a team for each long system and no more
        _check(batch, xs, res, precision)
        monkeypatch.setenv("XJPCG_BATCH_TEAMS", "0")
        st, ys, _ = h.batch_solve(batch, 20000, 1e-10, precision=precision)
        assert st == X.SUCCESS
        for x, y in zip(xs, ys):
            assert np.linalg.norm(x - y) <= 1e-8 * np.linalg.norm(y)
        assert h.check_guards()[1] == 0


def test_batched_input_errors_are_found_on_the_device(gpu_lib):
    batch = [_stencil((9, 10), k) for k in range(3)]
    with X.JPCG() as h:
        def call(rowptr, col, sysrow=None):
            n = np.cumsum([0] + [s.n for s in batch]).astype(np.int32) if sysrow is None else sysrow
            val, diag, b = (np.concatenate([getattr(s, f) for s in batch]) for f in ("val", "diag", "b"))
            x = np.zeros(270)
            st = h.lib.xJPCG_gbBatchSolve(h.h, 3, n.ctypes.data, rowptr.ctypes.data, col.ctypes.data, val.ctypes.data,
                                          diag.ctypes.data, b.ctypes.data, x.ctypes.data, 100, 1e-10, 0, None, 0)
            return st, h.last_message()
        off = np.cumsum([0] + [s.nnz for s in batch])
        rp = np.concatenate([[0]] + [s.rowptr[1:] + off[k] for k, s in enumerate(batch)]).astype(np.int32)
        col = np.concatenate([s.col for s in batch])
        for change, word in ((lambda r, c: r.__setitem__(0, 1), "start at 0"),
                             (lambda r, c: r.__setitem__(100, 0), "monotone"),
                             (lambda r, c: c.__setitem__(-1, 90), "column index"),
                             (lambda r, c: c.__setitem__(7, -1), "column index")):
            r, c = rp.copy(), col.copy()
            change(r, c)
            st, msg = call(r, c)
            assert st == X.INVALID_VALUE and word in msg, msg
        assert call(rp, col)[0] == X.SUCCESS


@pytest.mark.parametrize("precision", [0, 1])
def test_a_lost_post_ends_its_systems_alone(gpu_lib, precision, monkeypatch):
    # XJPCG_FAULT=post: in one iteration the last CTA of each cluster does not
    # post its sum to the first, whose wait then runs out (2 s).  The cluster gives
    # up as one and its system is reported as failed; systems of one CTA (at most
    # 128 rows) and the handle itself are as before.
    monkeypatch.setenv("XJPCG_FAULT", "post")
    monkeypatch.setenv("XJPCG_GUARD_BYTES", "4096")
    many = [_stencil((10, 11), k) for k in range(400)] + [_stencil((46, 47), 6), _stencil((25, 26, 27), 10)]
    with X.JPCG() as h:
        st, xs, res = h.batch_solve(many, 20000, 1e-10, precision=precision)
        assert st == X.EXECUTION_FAILED
        assert h.info().batchSmemRows == 0  # solved from shared memory
        assert [int(r["status"]) for r in res] == [0] * 400 + [2, 2]
        _check(many[:8], xs[:8], res[:8], precision)
        # ended in fewer iterations than the dropped one: nothing is lost
        st, _, res = h.batch_solve(many[-2:], 1, 1e-10, precision=precision)
        assert [int(r["status"]) for r in res] == [0, 0]
        assert h.check_guards()[1] == 0


@pytest.mark.parametrize("place", ["device", "misaligned", "pinned", "host"])
def test_batched_arrays_wherever_they_lie(gpu_lib, place):
    # only arrays of the handle's own device, aligned to their elements, are read
    # in place; everything else that a copy reaches is copied first (memory of
    # another device among it, which needs a second one to show)
    import torch
    batch = [_stencil((9, 10), 1), _stencil((25, 26), 2), _stencil((9, 10, 11), 3)]
    off = np.cumsum([0] + [s.nnz for s in batch])
    sys = np.cumsum([0] + [s.n for s in batch]).astype(np.int32)
    rp = np.concatenate([[0]] + [s.rowptr[1:] + off[k] for k, s in enumerate(batch)]).astype(np.int32)
    arrays = [rp] + [np.concatenate([getattr(s, f) for s in batch]) for f in ("col", "val", "diag", "b")]

    def put(a):
        t = torch.from_numpy(a)
        if place == "misaligned":
            raw = torch.zeros(a.nbytes + 1, dtype=torch.uint8, device="cuda")
            raw[1:] = torch.from_numpy(a.view(np.uint8)).cuda()
            return raw[1:]
        return t.cuda() if place == "device" else t.pin_memory() if place == "pinned" else t

    held = [put(a) for a in arrays]
    first, x = torch.from_numpy(sys).cuda(), torch.zeros(int(sys[-1]), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with X.JPCG() as h:
        st = h.lib.xJPCG_gbBatchSolve(h.h, 3, first.data_ptr(), *[t.data_ptr() for t in held], x.data_ptr(), 2000, 1e-10,
                                      0, None, 1)
        assert st == X.SUCCESS, h.last_message()
        _, want, _ = h.batch_solve(batch, 2000, 1e-10)
    assert np.array_equal(x.cpu().numpy(), np.concatenate(want))


@pytest.mark.parametrize("precision", [0, 1])
def test_batches_and_solves_without_clusters(gpu_lib, precision, monkeypatch):
    # a device that cannot hold a cluster (XJPCG_FAULT=cluster: the question is answered
    # with no): the kernels that need none run instead, in a forced form too
    monkeypatch.setenv("XJPCG_FAULT", "cluster")
    batch = BATCHES["clusters"]()
    with X.JPCG() as h:
        for teams in ("-1", "1"):
            monkeypatch.setenv("XJPCG_BATCH_TEAMS", teams)
            st, xs, res = h.batch_solve(batch, 20000, 1e-10, precision=precision)
            assert st == X.SUCCESS, h.last_message()
            assert h.info().batchSmemRows > 0 and h.info().batchGrid <= len(batch)  # one CTA per system
            _check(batch, xs, res, precision)
        s = batch[1]
        r = h.csr_solve(s.n, s.rowptr, s.col, s.val, s.diag, s.b, 20000, 1e-10)
        assert r.status == X.SUCCESS and oracle.true_relres(s.rowptr, s.col, s.val, s.b, r.x) <= 1.5e-10
