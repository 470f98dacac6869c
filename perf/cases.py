"""What a program that uses lap_gb300 has it do, at the sizes it does it.

A case is one call (or one training step) through the public entry points:
the solves behind gb_pcg_solve in each preconditioner and precision mode that
is used in earnest, LAP's own cg(), the adjoint, many systems and many
right-hand sides in one launch, the matrix-vector product, and the Matrix
Market reader.  Systems are the workloads of ``lap_gb300.gen`` (grids with
unit, lognormal and anisotropic weights, Chung-Lu power-law graphs, kNN
graphs), made from the seed; grids are built on the GPU and may have any
sides.  Right-hand sides are U[-1, 1] (the power-law graphs': N(0, 1)).

Tolerances are those of a solve whose x is wanted to nine digits or more,
whatever order the recurrence is rounded in: 1e-12, and 1e-10 on the
well-conditioned power-law graphs.
"""
import ctypes as C
import math

import numpy as np
import torch

import lap_gb300 as gb
from lap_gb300 import gen

MAXIT = 20000
SHIFT = {"unit": 1e-2, "lognormal": 1e-3, "aniso": 1e-2}


def listed():
    return [
        # LAP's own entry point on a small system, IC(0) data in pdata as its
        # driver leaves it: the call is launches, copies and latency
        dict(name="cg_ichol_20", kind="cg", nx=20, ny=20, nz=20, weights="lognormal", prec="ichol", tol=1e-12),
        # the 256 x 256 unit grid with line_jacobi, FP64: two kernels an
        # iteration, everything in L2
        dict(name="jacobi_256sq", kind="solve", nx=256, ny=256, nz=1, weights="unit", prec="line_jacobi",
             precision=0, tol=1e-12),
        # the benchmark's system, in its headline mode (FP32 operator and
        # preconditioner inside the FP64 recurrence)
        dict(name="ichol_split_128", kind="solve", nx=128, ny=128, nz=128, weights="lognormal", prec="ichol",
             precision=2, tol=1e-12),
        # the same system in the reference's precision
        dict(name="ichol_fp64_128", kind="solve", nx=128, ny=128, nz=128, weights="lognormal", prec="ichol",
             precision=0, tol=1e-12),
        # Gauss-Seidel on a box whose planes fit no tile size
        dict(name="gs_split_97x61x83", kind="solve", nx=97, ny=61, nz=83, weights="lognormal", prec="GS_std",
             precision=2, tol=1e-12),
        # one step of learning edge weights: forward solve, adjoint solve and
        # the gradients, on an anisotropic 2D grid
        dict(name="adjoint_1000x700", kind="adjoint", nx=1000, ny=700, nz=1, weights="aniso", prec="ichol",
             precision=2, tol=1e-12),
        # IC(0) on a power-law graph: hub rows, few levels, random numbering
        dict(name="powerlaw_fp64_128k", kind="powerlaw", n=1 << 17, graph=1003, prec="ichol", precision=0, tol=1e-10),
        # many small independent systems in one launch
        dict(name="batch_knn_48", kind="batch", count=48, nmin=1000, nmax=20000, graph=1004, prec="line_jacobi",
             precision=0, tol=1e-12),
        # 32 right-hand sides on one matrix
        dict(name="multi32_split_80", kind="multi", nx=80, ny=80, nz=80, weights="lognormal", nrhs=32,
             prec="line_jacobi", precision=2, tol=1e-12),
        # a nonlinear or time-stepping loop: new values on the old pattern,
        # refactor, solve
        dict(name="update_solve_64", kind="update", nx=64, ny=64, nz=64, weights="lognormal", prec="ichol",
             precision=2, tol=1e-12),
        # the product alone, as LAP's SpMV benchmark program calls it
        dict(name="spmv_128", kind="spmv", nx=128, ny=128, nz=128, weights="lognormal"),
        # a symmetric Matrix Market text in host memory into CSR on the device
        dict(name="mm_parse_60", kind="mm", nx=60, ny=60, nz=60),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cg", "jacobi", "ichol", "ichol", "ichol", "gs", "adjoint", "powerlaw", "batch", "multi",
                       "update", "spmv", "mm"])
    if kind == "cg":
        return dict(kind="cg", nx=_side(rng, 8, 48), ny=_side(rng, 8, 48), nz=_side(rng, 8, 48),
                    weights="lognormal", prec="ichol", tol=1e-12)
    if kind == "jacobi":
        return dict(kind="solve", nx=_side(rng, 32, 700), ny=_side(rng, 32, 700), nz=1, weights="unit",
                    prec="line_jacobi", precision=rng.choice([0, 0, 1]), tol=1e-12)
    if kind == "ichol":
        return dict(kind="solve", nx=_side(rng, 12, 128), ny=_side(rng, 12, 128), nz=_side(rng, 12, 128),
                    weights="lognormal", prec="ichol", precision=rng.choice([0, 1, 2, 2]), tol=1e-12)
    if kind == "gs":
        return dict(kind="solve", nx=_side(rng, 12, 110), ny=_side(rng, 12, 110), nz=_side(rng, 12, 110),
                    weights="lognormal", prec="GS_std", precision=rng.choice([0, 2]), tol=1e-12)
    if kind == "adjoint":
        return dict(kind="adjoint", nx=_side(rng, 60, 1000), ny=_side(rng, 60, 1000), nz=1, weights="aniso",
                    prec="ichol", precision=rng.choice([0, 2, 2]), tol=1e-12)
    if kind == "powerlaw":
        return dict(kind="powerlaw", n=_side(rng, 1 << 11, 1 << 17), graph=rng.randint(1, 9999), prec="ichol",
                    precision=rng.choice([0, 0, 2]), tol=1e-10)
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(4, 48), nmin=_side(rng, 100, 1000), nmax=_side(rng, 2000, 20000),
                    graph=rng.randint(1, 9999), prec="line_jacobi", precision=rng.choice([0, 2]), tol=1e-12)
    if kind == "multi":
        return dict(kind="multi", nx=_side(rng, 12, 64), ny=_side(rng, 12, 64), nz=_side(rng, 12, 64),
                    weights="lognormal", nrhs=rng.randint(2, 40), prec="line_jacobi", precision=rng.choice([0, 2]),
                    tol=1e-12)
    if kind == "update":
        return dict(kind="update", nx=_side(rng, 12, 90), ny=_side(rng, 12, 90), nz=_side(rng, 12, 90),
                    weights="lognormal", prec="ichol", precision=rng.choice([0, 2, 2]), tol=1e-12)
    if kind == "spmv":
        return dict(kind="spmv", nx=_side(rng, 12, 128), ny=_side(rng, 12, 128), nz=_side(rng, 12, 128),
                    weights="lognormal")
    return dict(kind="mm", nx=_side(rng, 8, 60), ny=_side(rng, 8, 60), nz=_side(rng, 8, 60))


# ------------------------------------------------------------------ inputs
def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _grid_edges(case, g):
    """Edge weights (x, y, z direction) of the grid, z-major."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    shapes = [(nz, ny, nx - 1), (nz, ny - 1, nx), (nz - 1, ny, nx)]
    kind = case["weights"]

    def normal(s):
        return torch.randn(s, generator=g, device="cuda", dtype=torch.float64)

    if kind == "unit":
        return [torch.ones(s, device="cuda", dtype=torch.float64) for s in shapes]
    if kind == "aniso":
        return [torch.exp(normal(shapes[0])), 0.1 * torch.exp(normal(shapes[1])), torch.exp(normal(shapes[2]))]
    return [torch.exp(0.5 * normal(s)) for s in shapes]


def _slots(dims, edges, diag):
    """[n, 7] values, columns and presence of a grid's rows: z-, y-, x-, the
    diagonal, x+, y+, z+ (columns ascending)."""
    nx, ny, nz = dims
    wx, wy, wz = edges
    n = nx * ny * nz
    lo = [torch.zeros(nz, ny, nx, device="cuda", dtype=wx.dtype) for _ in range(3)]
    hi = [torch.zeros(nz, ny, nx, device="cuda", dtype=wx.dtype) for _ in range(3)]
    lo[0][:, :, 1:], hi[0][:, :, :-1] = wx, wx
    lo[1][:, 1:, :], hi[1][:, :-1, :] = wy, wy
    lo[2][1:, :, :], hi[2][:-1, :, :] = wz, wz
    d = diag(lo, hi)
    v = torch.stack([-lo[2], -lo[1], -lo[0], d, -hi[0], -hi[1], -hi[2]], dim=-1).reshape(n, 7)
    idx = torch.arange(n, device="cuda")
    x, y, z = idx % nx, (idx // nx) % ny, idx // (nx * ny)
    c = torch.stack([idx - nx * ny, idx - nx, idx - 1, idx, idx + 1, idx + nx, idx + nx * ny], dim=-1)
    m = torch.stack([z > 0, y > 0, x > 0, x >= 0, x < nx - 1, y < ny - 1, z < nz - 1], dim=-1)
    return v, c, m


def _grid_csr(case, g):
    shift = SHIFT[case["weights"]]
    v, c, m = _slots((case["nx"], case["ny"], case["nz"]), _grid_edges(case, g),
                     lambda lo, hi: lo[0] + lo[1] + lo[2] + hi[0] + hi[1] + hi[2] + shift)
    ia = torch.zeros(v.shape[0] + 1, device="cuda", dtype=torch.int64)
    ia[1:] = m.sum(1).cumsum(0)
    return ia.to(torch.int32), c[m].to(torch.int32), v[m]


def _uniform(shape, g):
    return 2.0 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) - 1.0


def _digits(v, width):
    """[L, width] decimal digits of v, most significant first."""
    p = torch.tensor([10 ** (width - 1 - k) for k in range(width)], device="cuda", dtype=torch.int64)
    return (v[:, None] // p) % 10


def _mm_text(case, seed):
    """A grid Laplacian's lower triangle as Matrix Market text, and its CSR:
    every value is an integer over 10^15 written with 15 decimals."""
    g = _rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    one = 10 ** 15
    e = [torch.randint(1, one, s, generator=g, device="cuda", dtype=torch.int64)
         for s in [(nz, ny, nx - 1), (nz, ny - 1, nx), (nz - 1, ny, nx)]]
    v, c, m = _slots((nx, ny, nz), e, lambda lo, hi: lo[0] + lo[1] + lo[2] + hi[0] + hi[1] + hi[2] + one // 1000)
    n = v.shape[0]
    row = torch.arange(n, device="cuda")[:, None].expand(n, 7)
    low = m.clone()
    low[:, 4:] = False
    r, q, w = row[low] + 1, c[low] + 1, v[low]
    cols, keep = [], []

    def put(block, mask=None):
        cols.append(block)
        keep.append(torch.ones_like(block, dtype=torch.bool) if mask is None else mask)

    def char(ch, mask=None):
        put(torch.full((r.shape[0], 1), ord(ch), device="cuda", dtype=torch.int64), mask)

    for i in (r, q):
        d = _digits(i, 8)
        put(d + 48, d.cumsum(1) > 0)
        char(" ")
    char("-", (w < 0)[:, None])
    put(_digits(w.abs() // one, 1) + 48)
    char(".")
    put(_digits(w.abs() % one, 15) + 48)
    char("\n")
    body = torch.cat(cols, 1)[torch.cat(keep, 1)].to(torch.uint8).cpu().numpy().tobytes()
    head = "%%%%MatrixMarket matrix coordinate real symmetric\n%d %d %d\n" % (n, n, r.shape[0])
    return head.encode() + body, v[m].to(torch.float64) / one


def _inputs(case, seed):
    kind, g = case["kind"], _rng(seed)
    if kind == "mm":
        text, a = _mm_text(case, seed)
        return dict(text=text, a=a)
    if kind == "powerlaw":
        # the graph is the case's, its weights U(0, 1] and b the seed's: A = 1.001 D - W
        A, _ = gen.chung_lu(case["n"], seed=case["graph"])
        ia, ja = torch.from_numpy(A.ia).cuda(), torch.from_numpy(A.ja).cuda()
        n = A.n
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), (ia[1:] - ia[:-1]).long())
        col = ja.long()
        low, up = (col < row).nonzero()[:, 0], (col > row).nonzero()[:, 0]
        w = 1.0 - torch.rand(low.numel(), generator=g, device="cuda", dtype=torch.float64)
        a = torch.empty(ja.numel(), device="cuda", dtype=torch.float64)
        a[low] = -w
        a[up[torch.argsort(col[up] * n + row[up])]] = -w  # the mirror of each lower entry
        on = col == row
        a[on] = 0.0
        a[on] = torch.from_numpy(-1.001 * np.add.reduceat(a.cpu().numpy(), A.ia[:-1])).cuda()
        return dict(ia=ia, ja=ja, a=a, b=torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
    if kind == "batch":
        mats, _ = gen.knn_batch(case["count"], case["nmin"], case["nmax"], seed=case["graph"])
        for M in mats:  # the case's graphs, each system's weights in the seed's units
            M.a *= float(torch.rand((), generator=g, device="cuda") + 0.5)
        return dict(mats=mats, b=_uniform((sum(M.n for M in mats),), g))
    ia, ja, a = _grid_csr(case, g)
    n = ia.numel() - 1
    d = dict(ia=ia, ja=ja, a=a)
    d["b"] = _uniform((case["nrhs"], n) if kind == "multi" else (n,), g)
    if kind == "solve" and case["weights"] == "unit":
        d["b"] -= d["b"].mean()
    if kind == "adjoint":
        d["target"] = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    if kind == "update":
        d["a_new"] = _grid_csr(case, g)[2]
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    s = dict(case=case, d=d)
    if kind == "mm":
        return s
    if kind == "batch":
        s["batch"] = gb.Batch(d.pop("mats"), case["prec"])
    elif kind == "cg":
        # LAP's driver: pdata with the IC(0) factor on A's pattern
        n, nnz = d["ia"].numel() - 1, d["ja"].numel()
        d["factor"] = d["a"].clone()
        torch.cuda.synchronize()
        gb.lib().initialize_ichol(n, nnz, gb.ptr(d["ia"]), gb.ptr(d["ja"]), gb.ptr(d["factor"]))
        p = gb.PData()
        p.n, p.m, p.k, p.prec_op = n, 1, 1, case["prec"].encode()
        p.ichol_vals = gb.ptr(d["factor"])
        s["pdata"] = p
        s["hist"] = np.zeros(MAXIT + 3)
    else:
        s["sys"] = gb.System(d["ia"], d["ja"], d["a"], case.get("prec", "none"))
    return s


def run(state):
    case, d = state["case"], state["d"]
    kind = case["kind"]
    if kind == "mm":
        ia, ja, a, _ = gb.read_mm_device(data=d["text"])
        return dict(ia=ia, ja=ja, a=a)
    if kind == "spmv":
        return state["sys"].spmv(d["b"])
    if kind == "cg":
        n, nnz = d["ia"].numel() - 1, d["ja"].numel()
        x = torch.zeros_like(d["b"])
        it, flag = C.c_int(), C.c_int()
        torch.cuda.synchronize()  # x is zero before the library's own stream reads it
        gb.lib().cg(n, float(nnz), gb.ptr(d["ia"]), gb.ptr(d["ja"]), gb.ptr(d["a"]), gb.ptr(x), gb.ptr(d["b"]),
                    case["tol"], C.byref(state["pdata"]), MAXIT, C.byref(it), C.byref(flag),
                    state["hist"].ctypes.data)
        return x
    opts = dict(tol=case["tol"], maxit=MAXIT, precision=case["precision"])
    if kind == "batch":
        return state["batch"].solve(d["b"], **opts)[0]
    if kind == "multi":
        return gb.solve_multi(state["sys"], d["b"], **opts)[0]
    if kind == "update":
        state["sys"].set_values(d["a_new"])
        return state["sys"].solve(d["b"], **opts)[0]
    if kind == "adjoint":
        x, _ = state["sys"].solve(d["b"], **opts)
        lam, G, edges, _ = state["sys"].adjoint(x, x - d["target"], **opts)
        return dict(x=x, lam=lam, G=G, edges=edges)
    return state["sys"].solve(d["b"], **opts)[0]


# ------------------------------------------------------------------ work
def _grid_size(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    return n, n + 2 * (3 * n - nx * ny - (nx + ny) * nz)


def work(case):
    """Bytes and operations of one pass.  A solve's are those of its
    iterations, about as many as these systems take (a recurrence has to read
    the matrix, and the factor's two triangles, once in each): values in the
    mode's width, 4-byte indices, and x, r, p, q read and written."""
    kind = case["kind"]
    if kind == "mm":
        n, nnz = _grid_size(case)
        return dict(bytes=34.0 * (nnz + n) / 2 + 12.0 * nnz + 4.0 * n, flops=0.0)
    if kind == "powerlaw":
        n, nnz, iters = case["n"], 15 * case["n"], 20
    elif kind == "batch":
        mean = (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
        n = case["count"] * mean
        nnz, iters = 11 * n, 230
    else:
        n, nnz = _grid_size(case)
        side = max(case["nx"], case["ny"], case["nz"])
        iters = {"unit": 1.2, "lognormal": 2.3, "aniso": 0.17}[case["weights"]] * side
        if case.get("prec") == "line_jacobi" and case["weights"] == "lognormal":
            iters *= 3
    if kind == "spmv":
        return dict(bytes=12.0 * nnz + 4.0 * n + 16.0 * n, flops=2.0 * nnz)
    wide = 4 if case.get("precision", 0) else 8
    factor = case["prec"] != "line_jacobi"
    vec = 8.0 * (8 + (2 if factor else 1))
    cols = case.get("nrhs", 1)
    matrix = (nnz * (2 if factor else 1) * (4.0 + wide) + 4.0 * n) * math.ceil(cols / 32)
    passes = iters * (2 if kind == "adjoint" else 1)
    b = passes * (matrix + cols * vec * n)
    f = passes * cols * (2.0 * nnz * (2 if factor else 1) + 12.0 * n)
    if kind == "adjoint":
        b += 8.0 * nnz * 1.5
    if kind == "update":
        b += 12.0 * nnz + 8.0 * nnz
    return dict(bytes=b, flops=f)


# ------------------------------------------------------------------ exact
def _solve64(A, b, diag):
    """A x = b for each column of b [n, S] by plain diagonally scaled CG in
    64 bits, restarted from the true residual until it no longer shrinks."""
    x = torch.zeros_like(b)
    norm = b.norm(dim=0)
    best = math.inf
    for _ in range(4):
        r = b - A @ x
        worst = float((r.norm(dim=0) / norm).max())
        if worst < 2e-15 or worst > 0.2 * best:
            break
        best = worst
        dx = torch.zeros_like(b)
        z = r / diag
        p, rz = z.clone(), (r * z).sum(0)
        stop = max(1e-14 / worst, 1e-13)
        r0 = r.norm(dim=0)
        for it in range(20000):
            q = A @ p
            pq = (p * q).sum(0)
            alpha = torch.where(pq > 0, rz / pq, torch.zeros_like(pq))
            dx += alpha * p
            r -= alpha * q
            if it % 25 == 24 and bool((r.norm(dim=0) <= stop * r0).all()):
                break
            z = r / diag
            new = (r * z).sum(0)
            beta = torch.where(rz > 0, new / rz, torch.zeros_like(rz))
            p = z + beta * p
            rz = new
        x += dx
    return x


def exact(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    if kind == "mm":
        return dict(ia=None, ja=None, a=d["a"])
    if kind == "batch":
        mats, off, noff = d["mats"], 0, 0
        ia, ja, a = [np.zeros(1, np.int64)], [], []
        for M in mats:
            ia.append(M.ia[1:].astype(np.int64) + noff)
            ja.append(M.ja.astype(np.int64) + off)
            a.append(M.a)
            off, noff = off + M.n, noff + M.nnz
        ia, ja, a = (torch.from_numpy(np.concatenate(v)).cuda() for v in (ia, ja, a))
    else:
        ia, ja, a = d["ia"].long(), d["ja"].long(), d["a_new"] if kind == "update" else d["a"]
    n = ia.numel() - 1
    A = torch.sparse_csr_tensor(ia, ja, a, size=(n, n))
    if kind == "spmv":
        return (A @ d["b"][:, None])[:, 0]
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), ia[1:] - ia[:-1])
    diag = torch.zeros(n, device="cuda", dtype=torch.float64)
    on = row == ja
    diag[row[on]] = a[on]
    b = d["b"].t().contiguous() if kind == "multi" else d["b"][:, None]
    x = _solve64(A, b, diag[:, None])
    if kind == "multi":
        return x.t().contiguous()
    x = x[:, 0]
    if kind != "adjoint":
        return x
    lam = _solve64(A, (x - d["target"])[:, None], diag[:, None])[:, 0]
    low = ja < row
    i, j = row[low], ja[low]
    return dict(x=x, lam=lam, G=-lam[row] * x[ja], edges=-(lam[i] - lam[j]) * (x[i] - x[j]))
