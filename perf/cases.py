"""The workloads that this library's speed is judged on.

Every case goes through a public entry point of the xJPCG C ABI (most through
their ``hpc_gb300.JPCG`` methods).  Sizes come from the library's own
workloads (``hpc_gb300/workloads.py``, the tests and ``bench.py``): 7-point and
27-point grids, the reference example's tridiagonal system, Zipf-row SPD
matrices, batches of small stencil systems, the 96^3 adjoint problem.  The
inputs are drawn on the GPU with the same distributions as there.

Operations ("op"):

first   a solve that brings its matrix along (MODE_DEFAULT), from host arrays
values  a solve with new values on a known pattern (MODE_KEEP_NZ_LAYOUT), from
        host arrays: one step of a time integration or a Newton iteration
keep    a solve with a known matrix and a new b (MODE_KEEP_MATRIX), host b
device  a solve with a known matrix, b and x in device memory, fp64
mixed   the same with the FP32/FP64 solver
spmv    y = A x with a known matrix, x and y in device memory
batch   many small independent systems in one call, arrays in device memory
adjoint one step of fitting conductances to observations: forward solve with
        new values, adjoint solve, gradient per edge; host arrays
"""
import math

import numpy as np
import torch

import hpc_gb300 as X

MAX_ITER = 20000


def listed():
    return [
        # The smallest call: a known small matrix, one right-hand side after another.
        {"name": "keep_grid7_16", "op": "keep", "matrix": "grid7", "nx": 16, "ny": 16, "nz": 16, "tol": 1e-10},
        # The 7-point 32^3 parity system, same use.
        {"name": "keep_grid7_32", "op": "keep", "matrix": "grid7", "nx": 32, "ny": 32, "nz": 32, "tol": 1e-10},
        # The reference example's system through its symmetric-CSC call, 1-based, matrix and all.
        {"name": "first_tridiag_65536", "op": "first", "matrix": "tridiag", "n": 65536, "tol": 1e-10},
        # New coefficients on a known pattern, odd extents, COO in no order.
        {"name": "values_grid27_75x50x43", "op": "values", "matrix": "grid27", "nx": 75, "ny": 50, "nz": 43,
         "shuffled": True, "tol": 1e-10},
        # A first solve of a medium system from row-major COO: set-up, tuning and solve.
        {"name": "first_grid27_96", "op": "first", "matrix": "grid27", "nx": 96, "ny": 96, "nz": 96,
         "shuffled": False, "tol": 1e-10},
        # A step of fitting a 7-point 96^3 diffusion problem.
        {"name": "adjoint_grid7_96", "op": "adjoint", "nx": 96, "ny": 96, "nz": 96, "tol": 1e-12},
        # The headline system, resident on the device.
        {"name": "device_grid27_160", "op": "device", "matrix": "grid27", "nx": 160, "ny": 160, "nz": 160,
         "tol": 1e-10},
        # The same system in mixed precision, to the tolerance that gradients ask for.
        {"name": "mixed_grid27_160", "op": "mixed", "matrix": "grid27", "nx": 160, "ny": 160, "nz": 160,
         "tol": 1e-12},
        # Irregular rows: random columns, Zipf row lengths.
        {"name": "device_zipf_2M", "op": "device", "matrix": "zipf", "n": 2000000, "tol": 1e-10},
        # The product alone on a smaller irregular matrix of odd size.
        {"name": "spmv_zipf_300007", "op": "spmv", "matrix": "zipf", "n": 300007},
        # Many independent small systems, in both precisions.
        {"name": "batch_fp64_1024", "op": "batch", "count": 1024, "lo": 200, "hi": 20000, "mixed": False,
         "tol": 1e-10},
        {"name": "batch_mixed_1024", "op": "batch", "count": 1024, "lo": 200, "hi": 20000, "mixed": True,
         "tol": 1e-10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extents(rng, lo, hi):
    """Three extents of a grid of about lo .. hi points, none alike as a rule."""
    side = _log_int(rng, lo, hi) ** (1.0 / 3.0)
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    nx, ny = max(4, round(side * a)), max(4, round(side * b))
    return {"nx": nx, "ny": ny, "nz": max(4, round(side / (a * b)))}


def draw(rng):
    op = rng.choice(["keep", "values", "first", "device", "mixed", "spmv", "batch", "adjoint"])
    if op == "batch":
        lo = rng.choice([100, 200, 1000])
        return {"op": op, "count": _log_int(rng, 60, 1000), "lo": lo, "hi": _log_int(rng, 2 * lo, 20000),
                "mixed": rng.random() < 0.5, "tol": 1e-10}
    if op == "adjoint":
        return {"op": op, **_extents(rng, 4000, 880000), "tol": 1e-12}
    kinds = {"keep": ["grid7", "grid27"], "values": ["grid7", "grid27"], "first": ["grid7", "grid27", "tridiag"],
             "device": ["grid7", "grid27", "zipf"], "mixed": ["grid7", "grid27"],
             "spmv": ["grid7", "grid27", "zipf"]}
    matrix = rng.choice(kinds[op])
    case = {"op": op, "matrix": matrix}
    if matrix == "zipf":
        case["n"] = _log_int(rng, 50000, 1900000)
    elif matrix == "tridiag":
        case["n"] = _log_int(rng, 3000, 400000)
    else:
        most = {"keep": 300000, "values": 600000, "first": 800000}.get(op, 3800000)
        least = {"device": 30000, "mixed": 30000, "spmv": 200000}.get(op, 3000)
        case.update(_extents(rng, least, most))
    if op in ("values", "first") and matrix != "tridiag":
        case["shuffled"] = rng.random() < 0.5
    if op != "spmv":
        case["tol"] = 1e-12 if op == "mixed" else 1e-10
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
_FACES = [d for d in ((z, y, x) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1))
          if abs(d[0]) + abs(d[1]) + abs(d[2]) == 1]
_BOX = [(z, y, x) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1) if (z, y, x) != (0, 0, 0)]


def _generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * (int(seed) + 1) + salt)


def _lognormal(sigma, n, gen):
    if sigma == 0.0:
        return torch.ones(n, dtype=torch.float64, device="cuda")
    return torch.exp(sigma * torch.randn(n, dtype=torch.float64, device="cuda", generator=gen))


def _uniform(n, gen):
    return 2.0 * torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) - 1.0


class _Csr:
    """A matrix on the GPU: CSR with local columns, row index per entry, diagonal, b."""

    def __init__(self, n, rows, cols, vals, diag, b):
        self.n, self.rows, self.cols, self.vals, self.diag, self.b = n, rows, cols, vals, diag, b
        counts = torch.bincount(rows, minlength=n)
        self.rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        torch.cumsum(counts, 0, out=self.rowptr[1:])


def _stencil(dims, offsets, sigma, ghost_sigma, shift, gen):
    """sum_e c_e (e_i - e_j)(e_i - e_j)^T + ghosts + shift I over one grid or several, one after another.

    dims: (Z, Y, X) of each grid, as a list; a grid with Z = 1 is two-dimensional.  Edge conductances are
    log-normal(0, sigma), and so are the Dirichlet ghosts (ghost_sigma) of neighbours outside the grid.
    """
    d = torch.tensor(dims, dtype=torch.int64)
    sizes = d.prod(1)
    starts = torch.cumsum(sizes, 0) - sizes
    n = int(sizes.sum())
    if len(dims) == 1:
        Z, Y, W = (int(v) for v in dims[0])
        at = torch.arange(n, device="cuda")
        flat = Z == 1
    else:
        of = torch.repeat_interleave(torch.arange(len(dims), device="cuda"), sizes.cuda())
        Z, Y, W = (d[:, k].cuda()[of] for k in range(3))
        at = torch.arange(n, device="cuda") - starts.cuda()[of]
        flat = Z == 1
    x, y, z = at % W, (at // W) % Y, at // (W * Y)
    S = len(offsets) + 1
    full = sorted(offsets + [(0, 0, 0)])  # lexicographic: ascending columns
    vals = torch.zeros((n, S), dtype=torch.float64, device="cuda")
    have = torch.zeros((n, S), dtype=torch.bool, device="cuda")
    step = [None] * S
    diag = torch.full((n,), float(shift), dtype=torch.float64, device="cuda")
    mine = torch.arange(n, device="cuda")

    def inside(o):
        ok = (x + o[2] >= 0) & (x + o[2] < W) & (y + o[1] >= 0) & (y + o[1] < Y)
        return ok & (z + o[0] >= 0) & (z + o[0] < Z)

    for k, o in enumerate(full):
        step[k] = (o[0] * Y + o[1]) * W + o[2]
        if o <= (0, 0, 0):
            continue
        ok = inside(o)
        src = mine[ok]
        dst = src + (step[k][ok] if isinstance(step[k], torch.Tensor) else step[k])
        c = _lognormal(sigma, src.numel(), gen)
        vals[src, k] = -c
        vals[dst, S - 1 - k] = -c
        have[src, k] = True
        have[dst, S - 1 - k] = True
        diag[src] += c
        diag[dst] += c
    for o in offsets:
        out = ~inside(o)
        if o[0] != 0:
            out = out & ~flat if isinstance(flat, torch.Tensor) else (out if not flat else torch.zeros_like(out))
        diag[out] += _lognormal(ghost_sigma, int(out.sum()), gen)
    mid = S // 2
    vals[:, mid] = diag
    have[:, mid] = True
    if isinstance(Z, int):
        cols = at[:, None] + torch.tensor(step, device="cuda")[None, :]
    else:
        cols = at[:, None] + torch.stack([s if isinstance(s, torch.Tensor) else torch.full_like(at, s) for s in step], 1)
    rows = mine[:, None].expand(n, S)[have]
    return _Csr(n, rows, cols[have], vals[have], diag, _uniform(n, gen))


def _zipf(n, gen, seed):
    """Random symmetric matrix with Zipf(1.8) row lengths in 4 .. 4096, made SPD by its diagonal, scaled on both sides."""
    length = np.clip(np.random.default_rng(seed).zipf(1.8, n), 4, 4096).astype(np.int64)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.from_numpy(length).cuda())
    cols = torch.randint(0, n, (rows.numel(),), device="cuda", generator=gen)
    keep = rows != cols
    key = torch.unique(torch.minimum(rows, cols)[keep] * n + torch.maximum(rows, cols)[keep])
    a, b = key // n, key % n
    w = torch.randn(key.numel(), dtype=torch.float64, device="cuda", generator=gen)
    scale = 10.0 ** (6.0 * torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) - 3.0)
    r, c = torch.cat([a, b, torch.arange(n, device="cuda")]), torch.cat([b, a, torch.arange(n, device="cuda")])
    order = torch.argsort(r * n + c)
    key = (r * n + c)[order]
    # row sums of |w| on the host, where their order is fixed
    ha, hb, hw = a.cpu().numpy(), b.cpu().numpy(), w.abs().cpu().numpy()
    diag = 1.01 * torch.from_numpy(np.bincount(ha, hw, minlength=n) + np.bincount(hb, hw, minlength=n)).cuda()
    diag = torch.where(diag <= 0, torch.ones_like(diag), diag)
    r, c = key // n, key % n
    v = torch.cat([w, w, diag])[order] * scale[r] * scale[c]
    return _Csr(n, r, c, v, diag * scale * scale, _uniform(n, gen))


def _near_grid(n, ndim):
    if ndim == 2:
        w = max(2, round(math.sqrt(n)))
        return (1, max(2, round(n / w)), w)
    w = max(2, round(n ** (1.0 / 3.0)))
    y = max(2, round(math.sqrt(n / w)))
    return (max(2, round(n / (w * y))), y, w)


def _batch_dims(case):
    """The grids of a batch: a property of the case, whatever the seed of the values."""
    rng = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    out = []
    for _ in range(case["count"]):
        size = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        out.append(_near_grid(size, 2 if rng.random() < 0.5 else 3))
    return out


def _system(case, seed):
    gen = _generator(seed)
    dims = [(case.get("nz"), case.get("ny"), case.get("nx"))]
    if case["op"] == "batch":
        return _stencil(_batch_dims(case), _FACES, 1.0, 1.0, 0.0, gen)
    if case["op"] == "adjoint":
        return _stencil(dims, _FACES, 1.0, 0.0, 0.0, gen)
    if case["matrix"] == "grid7":
        return _stencil(dims, _FACES, 0.0, 0.0, 1e-3, gen)
    if case["matrix"] == "grid27":
        return _stencil(dims, _BOX, 1.5, 1.5, 0.0, gen)
    if case["matrix"] == "zipf":
        return _zipf(case["n"], gen, seed)
    n = case["n"]  # tridiagonal, diagonal 2.2, off-diagonal 1.0
    i = torch.arange(n, device="cuda")
    r = torch.cat([i, i[1:], i[:-1]])
    c = torch.cat([i, i[:-1], i[1:]])
    order = torch.argsort(r * n + c)
    v = torch.cat([torch.full((n,), 2.2, dtype=torch.float64, device="cuda"),
                   torch.ones(2 * (n - 1), dtype=torch.float64, device="cuda")])[order]
    b = torch.randint(0, n, (n,), device="cuda", generator=gen)
    return _Csr(n, r[order], c[order], v, torch.full((n,), 2.2, dtype=torch.float64, device="cuda"),
                (b - n // 2).double() / 97.0)


def _pinned(t):
    """A pinned host copy, as a numpy array."""
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy()


def _coo(m, shuffled, gen, pinned):
    order = torch.randperm(m.rows.numel(), device="cuda", generator=gen) if shuffled else None
    host = _pinned if pinned else (lambda t: t.cpu().numpy())
    pick = (lambda t: t[order]) if shuffled else (lambda t: t)
    return (host(pick(m.rows).to(torch.int32)).view(np.uint32), host(pick(m.cols).to(torch.int32)).view(np.uint32),
            host(pick(m.vals)))


def _need(r):
    if r.status != X.SUCCESS:
        raise RuntimeError("solve failed: %s" % r.message)
    return r


def prepare(case, seed):
    m = _system(case, seed)
    gen = _generator(seed, 1)
    s = {"case": case, "n": m.n, "h": X.JPCG()}
    h, op = s["h"], case["op"]
    if op == "batch":
        off = torch.cumsum(torch.tensor([0] + [z * y * w for z, y, w in _batch_dims(case)]), 0)
        s.update(sys=off.to(torch.int32).cuda(), rowptr=m.rowptr.to(torch.int32), col=m.cols.to(torch.int32),
                 val=m.vals, diag=m.diag, b=m.b, x=torch.zeros_like(m.b),
                 res=np.zeros(case["count"], X.BATCH_RESULT_DTYPE))
        torch.cuda.synchronize()
        return s
    s["diag"], s["b"] = _pinned(m.diag), _pinned(m.b)
    s["x"] = torch.zeros(m.n, dtype=torch.float64, pin_memory=True).numpy()
    if op == "first" and case["matrix"] == "tridiag":
        lower = m.cols <= m.rows  # row-major lower triangle = column-major upper triangle of a symmetric matrix
        s["ridx"] = _pinned(m.cols[lower] + 1)
        per = torch.bincount(m.rows[lower], minlength=m.n)
        s["cptr"] = _pinned(torch.cat([torch.ones(1, dtype=torch.int64, device="cuda"), 1 + torch.cumsum(per, 0)]))
        s["val"] = _pinned(m.vals[lower])
        return s
    keeps = op in ("first", "values", "adjoint")
    s["row"], s["col"], s["val"] = _coo(m, bool(case.get("shuffled")), gen, keeps)
    if op == "first":
        return s
    # the matrix as the program has set it before: one call that stops at once
    h.coo_solve(m.n, s["row"], s["col"], s["val"], s["diag"], s["b"], 0, 1e-10, x=s["x"])
    if op == "adjoint":
        upper = m.cols > m.rows
        s["ei"], s["ej"] = _pinned(m.rows[upper].to(torch.int32)), _pinned(m.cols[upper].to(torch.int32))
        s["c"] = _pinned(-m.vals[upper])
        s["obs"] = _pinned(_uniform(m.n, gen))
        s["lam"], s["grad"] = np.zeros(m.n), np.zeros(s["ei"].size)
    if not keeps:
        del s["row"], s["col"], s["val"]
    if op in ("device", "mixed"):
        s["db"], s["ddiag"], s["dx"] = m.b, m.diag, torch.zeros_like(m.b)
        if op == "mixed":  # its own tuning belongs to the known matrix
            _mixed(s, 1, 1e-1)
    if op == "spmv":
        s["dx"], s["dy"] = m.b, torch.zeros_like(m.b)
    torch.cuda.synchronize()
    return s


def _mixed(s, max_iter, tol):
    return s["h"].mixed_solve(s["db"].data_ptr(), s["ddiag"].data_ptr(), max_iter, tol, x=s["dx"].data_ptr(),
                              on_device=True)


def run(s):
    case, h, n = s["case"], s["h"], s["n"]
    op, tol = case["op"], case.get("tol")
    if op == "keep":
        return _need(h.coo_solve(n, None, None, None, s["diag"], s["b"], MAX_ITER, tol, mode=X.MODE_KEEP_MATRIX,
                                 x=s["x"])).x
    if op == "first" and "cptr" in s:
        return _need(h.csc_sym_solve(n, s["ridx"], s["cptr"], s["val"], s["diag"], s["b"], MAX_ITER, tol,
                                     mode=X.MODE_DEFAULT | X.MODE_FORTRAN_INDEX, x=s["x"])).x
    if op == "first":
        return _need(h.coo_solve(n, s["row"], s["col"], s["val"], s["diag"], s["b"], MAX_ITER, tol, x=s["x"])).x
    if op == "values":
        return _need(h.coo_solve(n, s["row"], s["col"], s["val"], s["diag"], s["b"], MAX_ITER, tol,
                                 mode=X.MODE_KEEP_NZ_LAYOUT, x=s["x"])).x
    if op == "device":
        st, _, _ = h.solve_device(s["db"].data_ptr(), s["ddiag"].data_ptr(), s["dx"].data_ptr(), MAX_ITER, tol)
        if st != X.SUCCESS:
            raise RuntimeError("solve failed: %s" % h.last_message())
        return s["dx"]
    if op == "mixed":
        _need(_mixed(s, MAX_ITER, tol))
        return s["dx"]
    if op == "spmv":
        h.spmv(s["dx"].data_ptr(), s["dy"].data_ptr(), on_device=True)
        return s["dy"]
    if op == "batch":
        st = h.lib.xJPCG_gbBatchSolve(h.h, case["count"], s["sys"].data_ptr(), s["rowptr"].data_ptr(),
                                      s["col"].data_ptr(), s["val"].data_ptr(), s["diag"].data_ptr(),
                                      s["b"].data_ptr(), s["x"].data_ptr(), MAX_ITER, tol,
                                      1 if case["mixed"] else 0, s["res"].ctypes.data, 1)
        if st != X.SUCCESS:
            raise RuntimeError("batched solve failed: %s" % h.last_message())
        return s["x"], s["res"]["status"].astype(np.int32)
    _need(h.coo_solve(n, s["row"], s["col"], s["val"], s["diag"], s["b"], MAX_ITER, tol, mode=X.MODE_KEEP_NZ_LAYOUT,
                      x=s["x"]))
    st, lam, _, _, _ = h.adjoint(s["x"] - s["obs"], s["diag"], MAX_ITER, tol, lam=s["lam"])
    if st != X.SUCCESS:
        raise RuntimeError("adjoint solve failed: %s" % h.last_message())
    return s["x"], lam, h.edge_grad(s["ei"], s["ej"], s["c"], out=s["grad"])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _size(case):
    """(rows, stored entries), for a random matrix the expected ones."""
    if case["op"] == "batch":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        n = case["count"] * mean
        return n, 5.7 * n
    if case.get("matrix") == "tridiag":
        return case["n"], 3 * case["n"] - 2
    if case.get("matrix") == "zipf":
        return case["n"], 17.4 * case["n"]
    x, y, z = case["nx"], case["ny"], case["nz"]
    if case.get("matrix") == "grid27":
        return x * y * z, (3 * x - 2) * (3 * y - 2) * (3 * z - 2)
    return x * y * z, x * y * z + 2 * ((x - 1) * y * z + x * (y - 1) * z + x * y * (z - 1))


def _iterations(case):
    """About how many iterations the tolerance takes (counts seen on these distributions)."""
    if case["op"] == "batch":
        return 317 * math.sqrt(case["hi"] / 20000)
    if case.get("matrix") == "tridiag":
        return 84
    if case.get("matrix") == "zipf":
        return 22
    side = (case["nx"] * case["ny"] * case["nz"]) ** (1.0 / 3.0)
    if case["op"] == "adjoint":
        return 2 * 6.6 * side
    return (3.6 if case["matrix"] == "grid27" else 3.2) * side * (1.2 if case["tol"] < 1e-11 else 1.0)


ON_CHIP = 200e6  # L2, registers and shared memory: a larger matrix has to be read again in every iteration


def work(case):
    n, nnz = _size(case)
    if case["op"] == "spmv":
        return {"bytes": 8 * nnz + 16 * n, "flops": 2 * nnz}
    k = _iterations(case)
    width = 4 if case["op"] == "mixed" or case.get("mixed") else 8
    index = {"first": 8, "batch": 4}.get(case["op"], 0)
    given = (8 + index) * nnz if case["op"] in ("first", "values", "adjoint", "batch") else width * nnz
    again = width * nnz * (k - 1) if width * nnz > ON_CHIP and case["op"] != "batch" else 0
    return {"bytes": given + again + 24 * n, "flops": k * (2 * nnz + 13 * n)}


# ---------------------------------------------------------------------------
# The same results in plain 64-bit torch
# ---------------------------------------------------------------------------
def _solve64(m, b):
    """A^-1 b by Jacobi-scaled CG in float64 until its residual stops falling."""
    root = torch.sqrt(m.diag)
    a = torch.sparse_csr_tensor(m.rowptr, m.glob, m.vals / (root[m.rows] * root[m.glob]), size=(m.n, m.n))
    rhs = b / root
    x = torch.zeros_like(rhs)
    for _ in range(3):  # twice restarted from the true residual
        r = rhs - torch.mv(a, x)
        p, rr = r.clone(), torch.dot(r, r)
        stop = 1e-30 * float(torch.dot(rhs, rhs))
        for k in range(6000):
            ap = torch.mv(a, p)
            alpha = rr / torch.dot(p, ap)
            x.add_(alpha * p)
            r.sub_(alpha * ap)
            new = torch.dot(r, r)
            p.mul_(new / rr).add_(r)
            rr = new
            if k % 25 == 24 and float(rr) <= stop:
                break
    return x / root


def exact(case, seed):
    m = _system(case, seed)
    m.glob = m.cols
    if case["op"] == "batch":
        sizes = torch.tensor([z * y * w for z, y, w in _batch_dims(case)])
        first = (torch.cumsum(sizes, 0) - sizes).cuda()
        of = torch.repeat_interleave(torch.arange(case["count"], device="cuda"), sizes.cuda())
        m.glob = m.cols + first[of][m.rows]
        return _solve64(m, m.b), None
    if case["op"] == "spmv":
        return torch.mv(torch.sparse_csr_tensor(m.rowptr, m.cols, m.vals, size=(m.n, m.n)), m.b)
    x = _solve64(m, m.b)
    if case["op"] != "adjoint":
        return x
    lam = _solve64(m, x - _uniform(m.n, _generator(seed, 1)))
    upper = m.cols > m.rows
    i, j = m.rows[upper], m.cols[upper]
    return x, lam, m.vals[upper] * (lam[i] - lam[j]) * (x[i] - x[j])
