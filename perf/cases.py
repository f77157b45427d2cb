"""The performance cases: what programs have this library do, call by call.

Every case builds its plan (or plans) once, as a program does before its
solver or training loop, and then times the call of the loop.  The matrices
are the workloads' kinds (grid Laplacians, power-law graphs, 27-point stencils
with coupled unknowns, uniform rows, bands), made from the seed on the GPU.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir,
                                "cb-sparse-dcu_b200"))
import cbspmv  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # an iterative solver's product on a grid small enough that the call
        # itself is the cost (coarse multigrid levels, test problems)
        dict(name="lap32_f64", kind="solve", matrix="lap", nx=32, ny=32, dtype="f64"),
        # the same on the 256 x 256 benchmark grid
        dict(name="lap256_f64", kind="solve", matrix="lap", nx=256, ny=256, dtype="f64"),
        # products with a scattered power-law matrix larger than the L2
        dict(name="pl_f64", kind="solve", matrix="pl", n=1048576, mean=16, dtype="f64"),
        # ... in FP32, at a size that fits no tile
        dict(name="pl_f32", kind="solve", matrix="pl", n=300007, mean=16, dtype="f32"),
        # a graph's adjacency matrix: every value 1, as Matrix Market pattern
        # files are read (PageRank, label propagation)
        dict(name="pl_unit_f64", kind="solve", matrix="pl", n=262147, mean=16, dtype="f64",
             unit=True),
        # a finite-element stiffness matrix, three unknowns a node
        dict(name="st_f64", kind="solve", matrix="st", g=32, dtype="f64"),
        # ... in FP32 with 32 x 32 blocks
        dict(name="st_f32_bs32", kind="solve", matrix="st", g=25, dtype="f32", bs=32),
        # features of a graph: 8 right-hand sides, FP32
        dict(name="pl_f32_rhs8", kind="block", matrix="pl", n=200003, mean=24, dtype="f32", rhs=8),
        # a block solver's product: 5 right-hand sides, FP64
        dict(name="uni_f64_rhs5", kind="block", matrix="uni", m=65537, n=65537, per_row=32,
             dtype="f64", rhs=5),
        # one training step's sparse layer: new values, forward, both gradients
        dict(name="train_f32_rhs8", kind="train", matrix="pl", n=100003, mean=24, graph=3,
             dtype="f32", rhs=8),
        # many uneven systems in one launch
        dict(name="batch_f32", kind="batch", count=32, nmin=1024, nmax=32768, mix=4, dtype="f32"),
        # least squares: A x, then A^T of it, on a tall matrix
        dict(name="normal_f64", kind="normal", matrix="uni", m=120011, n=50021, per_row=20,
             dtype="f64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lap", "pl", "pl", "unit", "st", "block", "block", "train", "batch",
                       "normal"])
    dtype = rng.choice(["f64", "f32"])
    if kind == "lap":
        return dict(kind="solve", matrix="lap", nx=_log(rng, 20, 600), ny=_log(rng, 20, 600),
                    dtype=dtype)
    if kind == "pl":
        return dict(kind="solve", matrix="pl", n=_log(rng, 4000, 400000),
                    mean=rng.randint(6, 20), dtype=dtype)
    if kind == "unit":
        return dict(kind="solve", matrix="pl", n=_log(rng, 4000, 260000),
                    mean=rng.randint(6, 20), dtype=dtype, unit=True)
    if kind == "st":
        return dict(kind="solve", matrix="st", g=_log(rng, 6, 32), dtype=dtype,
                    bs=rng.choice([16, 32]))
    if kind == "block":
        if rng.random() < 0.5:
            return dict(kind="block", matrix="pl", n=_log(rng, 4000, 160000),
                        mean=rng.randint(8, 24), dtype=dtype, rhs=rng.randint(2, 16))
        n = _log(rng, 4000, 100000)
        return dict(kind="block", matrix="uni", m=n, n=n, per_row=rng.randint(4, 40),
                    dtype=dtype, rhs=rng.randint(2, 16))
    if kind == "train":
        return dict(kind="train", matrix="pl", n=_log(rng, 4000, 100000),
                    mean=rng.randint(8, 24), graph=rng.randint(0, 10**6), dtype="f32",
                    rhs=rng.randint(1, 16))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(8, 32), nmin=1024, nmax=_log(rng, 2048, 32768),
                    mix=rng.randint(0, 10**6), dtype=dtype)
    return dict(kind="normal", matrix="uni", m=_log(rng, 4000, 120000),
                n=_log(rng, 4000, 120000), per_row=rng.randint(4, 24), dtype=dtype)


# ---- matrices (row-sorted COO on the GPU, no duplicates) -------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _unique(rows, cols, n):
    key = torch.unique(rows * n + cols)  # sorted
    return key // n, key % n


def _laplacian(nx, ny):
    i = torch.arange(nx * ny, device=DEV)
    x, y = i % nx, i // nx
    cols = torch.stack([i - nx, i - 1, i, i + 1, i + nx], 1)
    ok = torch.stack([y > 0, x > 0, x >= 0, x < nx - 1, y < ny - 1], 1)
    vals = torch.full((nx * ny, 5), -1.0, device=DEV, dtype=torch.float64)
    vals[:, 2] = 4.0
    rows = i[:, None].expand(-1, 5)
    return nx * ny, nx * ny, rows[ok], cols[ok], vals[ok]


def _lengths(n, mean, kmax, g):
    """Row lengths of a power law with exponent 2.1 on [1, kmax], shifted so
    that they have the mean asked for."""
    k = np.arange(1, kmax + 1, dtype=np.float64)
    lo, hi = -0.99, 1000.0
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        w = (k + mid) ** -2.1
        lo, hi = (mid, hi) if (w * k).sum() / w.sum() < mean else (lo, mid)
    cdf = torch.from_numpy(np.cumsum(w / w.sum())).to(DEV)
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    return (torch.searchsorted(cdf, u, right=True) + 1).clamp(max=kmax)


def _power_law(n, mean, g, band=4096):
    """70% of the columns near the diagonal, 30% anywhere."""
    lengths = _lengths(n, mean * 1.065, min(20000, n), g)
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), lengths)
    t = rows.numel()
    lo, hi = (rows - band).clamp(min=0), (rows + band).clamp(max=n - 1)
    u = torch.rand(t, generator=g, device=DEV, dtype=torch.float64)
    near = lo + (u * (hi - lo + 1)).long()
    far = torch.randint(0, n, (t,), generator=g, device=DEV)
    cols = torch.where(torch.rand(t, generator=g, device=DEV) < 0.7, near, far)
    rows, cols = _unique(rows, cols, n)
    return n, n, rows, cols, torch.randn(rows.numel(), generator=g, device=DEV,
                                         dtype=torch.float64)


def _stencil(k, g, dof=3):
    """27 points on a k^3 grid with dense dof x dof couplings, diagonally
    dominant."""
    node = torch.arange(k ** 3, device=DEV)
    x, y, z = node % k, (node // k) % k, node // (k * k)
    d = torch.tensor([-1, 0, 1], device=DEV)
    dz, dy, dx = (t.reshape(-1) for t in torch.meshgrid(d, d, d, indexing="ij"))
    ok = torch.ones(k ** 3, 27, dtype=torch.bool, device=DEV)
    for c, e in ((x, dx), (y, dy), (z, dz)):
        p = c[:, None] + e[None, :]
        ok &= (p >= 0) & (p < k)
    nbr = node[:, None] + (dx + k * dy + k * k * dz)[None, :]
    f = torch.arange(dof, device=DEV)
    shape = (k ** 3, dof, 27, dof)
    rows = (node[:, None] * dof + f)[:, :, None, None].expand(shape)
    cols = (nbr[:, :, None] * dof + f)[:, None, :, :].expand(shape)
    keep = ok[:, None, :, None].expand(shape)
    rows, cols = rows[keep], cols[keep]
    n = k ** 3 * dof
    vals = torch.rand(rows.numel(), generator=g, device=DEV, dtype=torch.float64) * 2 - 1
    diag = rows == cols
    vals[diag] = torch.bincount(rows, minlength=n)[rows[diag]].double()
    return n, n, rows, cols, vals


def _uniform(m, n, per_row, g):
    rows = torch.repeat_interleave(torch.arange(m, device=DEV), per_row)
    cols = torch.randint(0, n, (m * per_row,), generator=g, device=DEV)
    rows, cols = _unique(rows, cols, n)
    return m, n, rows, cols, torch.randn(rows.numel(), generator=g, device=DEV,
                                         dtype=torch.float64)


def _banded(n, bw, g):
    i = torch.arange(n, device=DEV)
    cols = i[:, None] + torch.arange(-bw, bw + 1, device=DEV)[None, :]
    ok = (cols >= 0) & (cols < n)
    rows = i[:, None].expand(cols.shape)[ok]
    return n, n, rows, cols[ok], torch.randn(rows.numel(), generator=g, device=DEV,
                                             dtype=torch.float64)


def _matrix(case, g):
    kind = case["matrix"]
    if kind == "lap":
        m, n, r, c, v = _laplacian(case["nx"], case["ny"])
    elif kind == "pl":
        m, n, r, c, v = _power_law(case["n"], case["mean"], g)
    elif kind == "st":
        m, n, r, c, v = _stencil(case["g"], g)
    elif kind == "uni":
        m, n, r, c, v = _uniform(case["m"], case["n"], case["per_row"], g)
    else:
        m, n, r, c, v = _banded(case["n"], case["bw"], g)
    if case.get("unit"):
        v = torch.ones_like(v)
    return m, n, r, c, v.to(_dtype(case)).double()


def _batch_items(case):
    """The matrices of a batch: log-uniform sizes, banded, power-law or
    uniform rows, 1 to 16 right-hand sides each."""
    rng = random.Random(case["mix"])
    items = []
    for _ in range(case["count"]):
        n, rhs = _log(rng, case["nmin"], case["nmax"]), rng.randint(1, 16)
        kind = rng.choice(["band", "pl", "uni"])
        it = dict(matrix=kind, n=n, rhs=rhs, dtype=case["dtype"])
        if kind == "band":
            it["bw"] = rng.randint(1, 64)
        elif kind == "pl":
            it["mean"] = 16
        else:
            it["m"] = n
            it["per_row"] = max(1, min(64, int(n * math.exp(rng.uniform(math.log(1e-4),
                                                                        math.log(1e-2))))))
        items.append(it)
    return items


def _dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _rand(g, dtype, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=dtype) * 2 - 1


# ---- the calls ---------------------------------------------------------------


def _plan(mat, case, **opts):
    m, n, r, c, v = mat
    plan = cbspmv.Plan(m=m, n=n, row=r.int().cpu().numpy(), col=c.int().cpu().numpy(),
                       val=v.cpu().numpy(), block_size=case.get("bs", 16),
                       value_type=cbspmv.F64 if case["dtype"] == "f64" else cbspmv.F32, **opts)
    return plan.upload()


def _inputs(case, seed):
    """The matrix (or matrices) and the vectors of a case."""
    g, dt = _gen(seed), _dtype(case)
    if case["kind"] == "batch":
        items = _batch_items(case)
        mats = [_matrix(it, g) for it in items]
        return mats, [_rand(g, dt, a[1], it["rhs"]) for a, it in zip(mats, items)]
    # a training run keeps its graph: that comes with the case, the values,
    # features and targets with the seed
    mat = _matrix(case, _gen(case["graph"]) if "graph" in case else g)
    shape = (mat[1], case["rhs"]) if case.get("rhs", 1) > 1 else (mat[1],)
    x = _rand(g, dt, *shape)
    if case["kind"] == "train":
        target = torch.randn((mat[0],) + shape[1:], generator=g, device=DEV, dtype=dt)
        vals = torch.randn(mat[2].numel(), generator=g, device=DEV, dtype=dt)
        return mat, x, target, vals
    return mat, x


def prepare(case, seed):
    kind = case["kind"]
    inputs = _inputs(case, seed)
    if kind == "batch":
        mats, xs = inputs
        items = _batch_items(case)
        plans = [_plan(a, case) for a in mats]
        ys = [torch.empty(a[0], it["rhs"], dtype=x.dtype, device=DEV)
              for a, it, x in zip(mats, items, xs)]
        batch = cbspmv.Batch(plans, [it["rhs"] for it in items]).bind(xs, ys)
        return dict(kind=kind, batch=batch, ys=ys)
    if kind == "train":
        mat, x, target, vals = inputs
        plan = _plan(mat, case, want_transpose=1)
        return dict(kind=kind, plan=plan, x=x.requires_grad_(), vals=vals.requires_grad_(),
                    target=target)
    mat, x = inputs
    plan = _plan(mat, case, want_transpose=int(kind == "normal"))
    s = dict(kind=kind, plan=plan, x=x)
    if kind != "block":  # a solver's loop keeps its vectors
        s["y"] = torch.empty(mat[0], dtype=x.dtype, device=DEV)
    if kind == "normal":
        s["z"] = torch.empty(mat[1], dtype=x.dtype, device=DEV)
    return s


def run(s):
    kind = s["kind"]
    if kind == "solve":
        return s["plan"].spmv(s["x"], s["y"])
    if kind == "block":
        return s["plan"].spmv(s["x"])
    if kind == "normal":
        y = s["plan"].spmv(s["x"], s["y"])
        return y, s["plan"].spmv_t(y, s["z"])
    if kind == "train":  # loss 0.5 |Y - T|^2
        y = cbspmv.cbspmv_apply(s["plan"], s["vals"], s["x"])
        gv, gx = torch.autograd.grad(y, (s["vals"], s["x"]), y.detach() - s["target"])
        return y.detach(), gv, gx
    s["batch"].run()
    return s["ys"]


# ---- what they are held to ---------------------------------------------------


def _mul(rows, cols, vals, x, m):
    x = x.double()
    one = x.dim() == 1
    x = x[:, None] if one else x
    y = torch.stack([torch.zeros(m, device=DEV, dtype=torch.float64).index_add_(
        0, rows, vals * x[cols, j]) for j in range(x.shape[1])], 1)
    return y[:, 0] if one else y


def exact(case, seed):
    inputs = _inputs(case, seed)
    kind = case["kind"]
    if kind == "batch":
        return [_mul(r, c, v, x, m) for (m, n, r, c, v), x in zip(*inputs)]
    if kind == "train":
        (m, n, r, c, _), x, target, vals = inputs
        vals, x = vals.double(), x.double()
        y = _mul(r, c, vals, x, m)
        d = y - target.double()
        if x.dim() == 1:
            gv = d[r] * x[c]
        else:
            gv = sum(d[r, j] * x[c, j] for j in range(x.shape[1]))
        return y, gv, _mul(c, r, vals, d, n)
    (m, n, r, c, v), x = inputs
    y = _mul(r, c, v, x, m)
    return (y, _mul(c, r, v, y, n)) if kind == "normal" else y


def _size(case):
    """Rows, columns and (expected) entries."""
    kind = case["matrix"]
    if kind == "lap":
        nx, ny = case["nx"], case["ny"]
        return nx * ny, nx * ny, 5 * nx * ny - 2 * (nx + ny)
    if kind == "pl":
        return case["n"], case["n"], case["n"] * case["mean"]
    if kind == "st":
        n = 3 * case["g"] ** 3
        return n, n, 9 * (3 * case["g"] - 2) ** 3
    if kind == "uni":
        return case["m"], case["n"], case["m"] * case["per_row"]
    n, bw = case["n"], case["bw"]
    return n, n, n * (2 * bw + 1) - bw * (bw + 1)


def work(case):
    """An index of 4 bytes and a value per entry, each vector once."""
    if case["kind"] == "batch":
        per = [work(dict(it, kind="block")) for it in _batch_items(case)]
        return {k: sum(w[k] for w in per) for k in ("bytes", "flops")}
    m, n, nnz = _size(case)
    vsz = 8 if case["dtype"] == "f64" else 4
    entry = 4 + (0 if case.get("unit") else vsz)
    rhs = case.get("rhs", 1)
    nbytes, flops = nnz * entry + (m + n) * rhs * vsz, 2 * nnz * rhs
    if case["kind"] == "normal":
        nbytes, flops = 2 * nbytes, 2 * flops
    if case["kind"] == "train":  # forward, A^T G and the value gradient; X and Y - T again
        nbytes, flops = 2 * nbytes + nnz * vsz + (m + n) * rhs * vsz, 3 * flops
    return {"bytes": nbytes, "flops": flops}
