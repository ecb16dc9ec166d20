"""The workloads whose speed this library is judged by: nested F3R solves, and
the single operators a solve is made of, through the Python entry points.

A case is a dict of plain values.  `kind` says which entry point it goes
through:

  solve     Solver.solve, one right-hand side (with `host`: numpy vectors, which
            the call copies to the device and back)
  multi     Solver.solve_multi, several right-hand sides of one system
  batch     Batch.solve, several systems of one sparsity pattern
  operate   Sell.operate, out = A in
  residual  Sell.compute_residual, res = rhs - A in
  trsv      Trsv.solve, a triangular solve by Jacobi sweeps
  learned   Learned.evaluate(grad=True), loss and gradient of the network that
            corrects SDAINV's values (forward and backward)

The matrices are the ones the library generates: the 27-point stencil in the
reference generators' variants (0 hpcg, 1 hpgmp, 2 half-space nonsymmetric) and
7-point diffusion with log-normal coefficients; both diagonally scaled, as the
drivers do.  A matrix and its solver are set up once and serve every
right-hand side, as in a user's program; the seed draws the right-hand sides
(solutions U(-1, 1)), operands and network weights.
"""
import functools
import math

import numpy as np
import torch

import f3r_b200 as F
from f3r_b200.learned import Learned, block_diag

# storage layouts a caller chooses between
LAYOUTS = {
    "packed": dict(),                                                  # the library's default: SELL-32, sigma 1
    "sigma256": dict(sell_sigma=256),                                  # SELL-C-sigma as the configuration names it
    "aligned": dict(sell_align=1),                                     # offset-aligned 32-row slices
    "aligned64": dict(sell_align=1, sell_c=64),                        # offset-aligned 64-row slices (the benchmark's)
    "csr": dict(format=F.FORMAT_CSR),
}
SELL = {
    "packed": dict(),
    "sigma256": dict(sigma=256),
    "aligned": dict(aligned=True),
    "aligned64": dict(aligned=True, height=64),
    "csr": dict(csr=True),
}
NP = {"f64": np.float64, "f32": np.float32, "f16": np.float16}
TORCH = {"f64": torch.float64, "f32": torch.float32, "f16": torch.float16}
VAL = {"f64": F.F64, "f32": F.F32, "f16": F.F16}
SIZE = {"f64": 8, "f32": 4, "f16": 2}
TOL = 1e-10
FIELD = dict(sigma=1.5, corr_len=6.0)  # the learned configuration's coefficient fields


def listed():
    return [
        # the smallest call: a small system in the default layout, vectors on the host
        dict(name="solve-27pt-16", kind="solve", matrix="27pt", variant=2, nx=16, ny=16, nz=16, layout="packed",
             precond="sdainv", host=True),
        # the headline benchmark: 192^3 nonsymmetric 27-point stencil in the benchmark's layout
        dict(name="solve-27pt-192", kind="solve", matrix="27pt", variant=2, nx=192, ny=192, nz=192,
             layout="aligned64", precond="sdainv", host=False),
        # SELL-C-sigma with C = 32 and sigma = 256, as the configuration states it, on an odd box
        dict(name="solve-27pt-sigma256", kind="solve", matrix="27pt", variant=1, nx=95, ny=83, nz=71,
             layout="sigma256", precond="sdainv", host=False),
        # variable coefficients: the learned configuration's 128^3 field under plain SDAINV (general factors)
        dict(name="solve-7pt-128", kind="solve", matrix="7pt", variant=0, nx=128, ny=128, nz=128,
             layout="aligned64", precond="sdainv", host=False),
        # the reference's CPU configuration: 64^3, CSR, block-Jacobi ILU(0) over 112 blocks
        dict(name="solve-ilu-64", kind="solve", matrix="27pt", variant=0, nx=64, ny=64, nz=64, layout="csr",
             precond="ilu", host=True),
        # one system of the batched configuration (grid edges 16..112, 1..16 right-hand sides)
        dict(name="multi-27pt-81-7", kind="multi", matrix="27pt", variant=0, nx=81, ny=81, nz=81, layout="aligned",
             precond="sdainv", rhs=7),
        # systems of one pattern solved together (coefficient fields of one grid)
        dict(name="batch-7pt-48-8", kind="batch", matrix="7pt", variant=0, nx=48, ny=48, nz=48, layout="packed",
             precond="sdainv", systems=8),
        # level 3's product on a large variable-coefficient matrix (the precision-stress configuration's kind)
        dict(name="operate-f16-7pt-200", kind="operate", matrix="7pt", variant=0, nx=200, ny=200, nz=200,
             layout="aligned64", val="f16", vec="f32"),
        # level 2's product on a small system in CSR
        dict(name="operate-f32-27pt-40", kind="operate", matrix="27pt", variant=2, nx=40, ny=40, nz=40, layout="csr",
             val="f32", vec="f32"),
        # the outer fp64 residual, default layout, ragged box
        dict(name="residual-f64-27pt-101", kind="residual", matrix="27pt", variant=1, nx=101, ny=67, nz=59,
             layout="packed", val="f64", vec="f64"),
        # the reference GPU drivers' ILU solve: two Jacobi sweeps on the lower factor
        dict(name="trsv-jacobi-64", kind="trsv", matrix="27pt", variant=0, nx=64, ny=64, nz=64, iters=2),
        # training of the learned correction: 16 stacked 24^3 fields, 4 pairs
        dict(name="learned-grad-24", kind="learned", matrix="7pt", variant=0, nx=24, ny=24, nz=24, fields=16, pairs=4),
    ]


def draw(rng):
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def box(lo, hi):
        e = edge(lo, hi)
        return {k: max(lo, min(hi, int(e * rng.uniform(0.8, 1.2)))) for k in ("nx", "ny", "nz")}

    kind = rng.choice(["solve", "solve", "solve", "multi", "batch", "operate", "operate", "residual", "trsv", "learned"])
    matrix = rng.choice(["27pt", "7pt"])
    variant = rng.randrange(3) if matrix == "27pt" else 0
    layout = rng.choice(["packed", "sigma256", "aligned", "aligned64", "csr"])
    c = dict(kind=kind, matrix=matrix, variant=variant, layout=layout)
    if kind == "solve":
        if rng.random() < 0.25:  # block-Jacobi ILU(0) in the reference's two storages
            return dict(c, **box(24, 80), matrix="27pt", variant=rng.randrange(2), precond="ilu",
                        layout=rng.choice(["csr", "packed"]), host=rng.random() < 0.5)
        return dict(c, **box(32 if layout == "aligned64" else 14, 128), precond="sdainv", host=rng.random() < 0.3)
    if kind == "multi":
        return dict(c, **box(32 if layout == "aligned64" else 16, 96), precond="sdainv", rhs=rng.randint(2, 16))
    if kind == "batch":
        return dict(c, **box(16, 56), matrix="7pt", variant=0, layout="packed", precond="sdainv",
                    systems=rng.randint(2, 12))
    if kind == "operate":
        val, vec = rng.choice([("f64", "f64"), ("f32", "f32"), ("f16", "f32"), ("f16", "f16")])
        return dict(c, **box(32 if layout == "aligned64" else 16, 160), val=val, vec=vec)
    if kind == "residual":
        t = rng.choice(["f64", "f32", "f16"])
        return dict(c, **box(32 if layout == "aligned64" else 16, 160), val=t, vec=t)
    if kind == "trsv":
        return dict(kind=kind, matrix="27pt", variant=0, **box(24, 96), iters=rng.randint(1, 4))
    e = rng.randint(12, 28)
    return dict(kind="learned", matrix="7pt", variant=0, nx=e, ny=e, nz=e, fields=rng.randint(4, 24),
                pairs=rng.randint(2, 8))


# ---- set-up that a user's program keeps -------------------------------------

@functools.lru_cache(maxsize=1)
def _context():
    return F.Context(0)


def _matrix(case, field=0):
    n3 = case["nx"], case["ny"], case["nz"]
    if case["matrix"] == "27pt":
        return F.stencil27(*n3, case["variant"], 0.5).scale()
    return F.diffusion7(*n3, **FIELD, seed=field).scale()


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "host")))


@functools.lru_cache(maxsize=1)
def _setup(key):
    """The matrices of a case and the object that works on them."""
    case, ctx = dict(key), _context()
    kind = case["kind"]
    if kind in ("solve", "multi", "batch"):
        kw = dict(rel_tol=TOL, **LAYOUTS[case["layout"]])
        if case["precond"] == "ilu":
            kw.update(precond=F.PRECOND_ILU0_BJ, max_restarts=3)
        if kind == "batch":
            mats = [_matrix(case, f) for f in range(case["systems"])]
            return mats, F.Batch(ctx, mats, **kw)
        A = _matrix(case)
        return [A], F.Solver(ctx, A, **kw)
    if kind in ("operate", "residual"):
        A = _matrix(case)
        return [A], F.Sell(ctx, A, dtypes=(VAL[case["val"]],), **SELL[case["layout"]])
    if kind == "trsv":
        L, _ = _matrix(case).ilu0_bj(blocks=112)
        return [L], F.Trsv(ctx, L, F.TRSV_LOWER, F.TRSV_JACOBI, case["iters"], 1.0)
    A = block_diag([_matrix(case, f) for f in range(case["fields"])])
    Z, Wt = A.sdainv()
    return [A, Z, Wt], None


def _solutions(case, n, seed):
    r = np.random.default_rng(seed)
    k = case.get("rhs", case.get("systems", case.get("pairs", 1)))
    return r.uniform(-1.0, 1.0, (k, n))


def _weights(seed):
    """Network weights of a trained network's size: He-normal hidden layers, a small output layer."""
    r = np.random.default_rng(seed + 7919)
    return np.concatenate([r.normal(0, math.sqrt(2 / 7), 448), r.normal(0, 0.05, 64),
                           r.normal(0, math.sqrt(2 / 64), 4096), r.normal(0, 0.05, 64),
                           r.normal(0, 0.02, 512), r.normal(0, 0.01, 8)]).astype(np.float32)


def prepare(case, seed):
    mats, obj = _setup(_key(case))
    kind, n = case["kind"], mats[0].shape[0]
    if kind in ("solve", "multi", "batch"):
        xs = _solutions(case, n, seed)
        b = np.stack([mats[min(i, len(mats) - 1)].spmv(x) for i, x in enumerate(xs)])
        if kind == "solve":
            b = b[0]
        b = b if case.get("host") else torch.from_numpy(b).cuda()
        return dict(kind=kind, solver=obj, b=b)
    if kind == "learned":
        e = _solutions(case, n, seed)
        net = Learned(_context())
        net.params = _weights(seed)
        net.set_data(mats[0], case["nx"], case["ny"], mats[1], mats[2],
                     np.stack([mats[0].spmv(x) for x in e]), e)
        return dict(kind=kind, net=net)
    vec = "f16" if kind == "trsv" else case["vec"]
    r = np.random.default_rng(seed)
    x = torch.from_numpy(r.uniform(-1.0, 1.0, n).astype(NP[vec])).cuda()
    st = dict(kind=kind, op=obj, x=x, y=torch.empty_like(x))
    if kind == "residual":
        st["b"] = torch.from_numpy(r.uniform(-1.0, 1.0, n).astype(NP[vec])).cuda()
    if kind in ("operate", "residual"):
        st["val"] = VAL[case["val"]]
    return st


def run(st):
    kind = st["kind"]
    if kind == "solve":
        b = st["b"]
        x = np.zeros_like(b) if isinstance(b, np.ndarray) else torch.zeros_like(b)
        r = st["solver"].solve(b, x)
        return {"x": x, "steps": r.res_iter}
    if kind == "multi":
        X = torch.zeros_like(st["b"])
        r = st["solver"].solve_multi(st["b"], X)
        return {"x": X, "steps": np.array([q.res_iter for q in r])}
    if kind == "batch":
        X = torch.zeros_like(st["b"])
        r = st["solver"].solve(list(st["b"]), list(X))
        return {"x": X, "steps": np.array([q.res_iter for q in r])}
    if kind == "operate":
        st["op"].operate(st["x"], st["y"], val_t=st["val"])
        return st["y"]
    if kind == "residual":
        st["op"].compute_residual(st["b"], st["x"], st["y"], val_t=st["val"])
        return st["y"]
    if kind == "trsv":
        st["op"].solve(st["x"], st["y"])
        return st["y"]
    loss, grad = st["net"].evaluate(grad=True)
    return {"loss": loss, "grad": grad}


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    row = 27 if case["matrix"] == "27pt" else 7
    nnz = row * n
    kind = case["kind"]
    if kind in ("operate", "residual"):
        s, v = SIZE[case["val"]], SIZE[case["vec"]]
        vecs = 3 if kind == "residual" else 2
        return {"bytes": nnz * (s + 4) + 4 * (n + 1) + vecs * v * n, "flops": 2 * nnz}
    if kind == "trsv":
        half = (nnz - n) // 2
        return {"bytes": half * 6 + 4 * (n + 1) + 4 * n, "flops": 2 * half * case["iters"]}
    if kind == "learned":
        rows = n * case["fields"]
        # forward and backward of 4,992 weights a row; features, factors and pairs read once
        return {"bytes": rows * (28 + 2 * 4 * 12 + case["pairs"] * 16) + 4 * 5192, "flops": 3 * 2 * 4992 * rows}
    # one outer step of each system and right-hand side: 64 fp16 products, 8 fp32 and one fp64, matrices in
    # CSR read once a product for all right-hand sides, the vectors of each
    systems, k = case.get("systems", 1), case.get("rhs", 1)
    matrix = systems * (64 * nnz * 6 + 8 * nnz * 8 + nnz * 12)
    vectors = systems * k * n * (64 * 4 + 8 * 8 + 16)
    return {"bytes": matrix + vectors, "flops": systems * k * 73 * 2 * nnz}


# ---- the same results in 64 bits, by plain torch --------------------------------

def _sparse(M, keep=None):
    r, i, v = M.arrays()
    rows = np.repeat(np.arange(len(r) - 1), np.diff(r))
    if keep is not None:
        m = keep(rows, i)
        rows, i, v = rows[m], i[m], v[m]
    at = torch.from_numpy(np.stack([rows, i.astype(np.int64)])).cuda()
    n = M.shape[0]
    return torch.sparse_coo_tensor(at, torch.from_numpy(v).cuda(), (n, n), is_coalesced=True).to_sparse_csr()


def _features(M, nx, ny):
    """Coefficients of every row at offsets 0, -1, +1, -nx, +nx, -nx ny, +nx ny."""
    r, i, v = M.arrays()
    rows = np.repeat(np.arange(len(r) - 1), np.diff(r))
    f = np.zeros((len(r) - 1, 7))
    for k, d in enumerate((0, -1, 1, -nx, nx, -nx * ny, nx * ny)):
        at = i - rows == d
        f[rows[at], k] = v[at]
    return torch.from_numpy(f).cuda()


def _corrected(M, offs, delta):
    """M's values times 1 + delta of their row and offset, as (rows, columns, values)."""
    r, i, v = M.arrays()
    rows = np.repeat(np.arange(len(r) - 1), np.diff(r))
    slot = np.full(len(i), -1)
    for k, d in enumerate(offs):
        slot[i - rows == d] = k
    at, col = torch.from_numpy(rows).cuda(), torch.from_numpy(i.astype(np.int64)).cuda()
    vt, st = torch.from_numpy(v).cuda(), torch.from_numpy(slot).cuda()
    d = delta[at, st.clamp(min=0)]
    return at, col, torch.where(st >= 0, vt * (1 + d), vt)


def _exact_gradient(case, mats, seed):
    A, Z, Wt = mats
    nx, sxy = case["nx"], case["nx"] * case["ny"]
    p = torch.from_numpy(_weights(seed).astype(np.float64)).cuda().requires_grad_()
    W1, b1, W2, b2, W3, b3 = torch.split(p, [448, 64, 4096, 64, 512, 8])
    h = torch.relu(_features(A, nx, case["ny"]) @ W1.view(64, 7).T + b1)
    h = torch.relu(h @ W2.view(64, 64).T + b2)
    delta = h @ W3.view(8, 64).T + b3
    e = _solutions(case, A.shape[0], seed)
    r = torch.from_numpy(np.stack([A.spmv(x) for x in e])).cuda()
    e = torch.from_numpy(e).cuda()

    def times(M, offs, d, x):
        at, col, v = _corrected(M, offs, d)
        return torch.zeros_like(x).index_add(1, at, v * x[:, col])

    y = times(Wt, (0, -1, -nx, -sxy), delta[:, 4:], r)
    y = times(Z, (0, 1, nx, sxy), delta[:, :4], y)
    loss = (((y - e) ** 2).sum(1) / (e ** 2).sum(1)).mean()
    loss.backward()
    return {"loss": loss.item(), "grad": p.grad}


def exact(case, seed):
    mats, _ = _setup(_key(case))
    kind, n = case["kind"], mats[0].shape[0]
    if kind in ("solve", "multi", "batch"):
        x = _solutions(case, n, seed)
        return {"x": x[0] if kind == "solve" else x, "steps": None}
    if kind == "learned":
        return _exact_gradient(case, mats, seed)
    r = np.random.default_rng(seed)
    vec = "f16" if kind == "trsv" else case["vec"]
    x = torch.from_numpy(r.uniform(-1.0, 1.0, n).astype(NP[vec]).astype(np.float64)).cuda()
    if kind == "trsv":  # unit lower factor: y = x, then sweeps y = x - N y
        N = _sparse(mats[0], lambda rows, cols: cols < rows)
        y = x
        for _ in range(case["iters"]):
            y = x - N @ y
        return y
    y = _sparse(mats[0]) @ x
    if kind == "operate":
        return y
    return torch.from_numpy(r.uniform(-1.0, 1.0, n).astype(NP[vec]).astype(np.float64)).cuda() - y
