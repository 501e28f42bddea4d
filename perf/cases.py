"""Performance cases of raptor_b200, through its public Python API.

Each case is one call sequence that a program using the library runs many
times: sparse products, an AMG setup, an AMG or AMG-PCG solve, several
right-hand sides or several systems at once, and a differentiated solve.
Operators are the gallery's (27-point Laplacian, rotated anisotropic
diffusion, 7-point anisotropic diffusion), finite-volume diffusion with a
smooth log-normal conductivity, unstructured CSR rows and block CSR.

    listed()              the named cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   inputs and handles a program holds before the call
    run(state)            one pass
    exact(case, seed)     the pass's outputs in FP64 by direct methods
    work(case)            bytes and operations a pass cannot do without
    tolerance(case)       how far two correct runs may be apart
"""
import ctypes
import math

import numpy as np
import torch

import raptor_b200 as rb

TOL = 1e-8           # true relative residual of the iterative solves
EPS, THETA = 0.001, math.pi / 8.0   # the rotated diffusion of the solves


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # the product family on the smallest operator of the examples (10,000
        # rows, 9-point): what a Krylov method written in Python calls
        {"name": "products_rot2d_100", "kind": "products", "op": "rot2d", "side": 100},
        # the same four products on a large stencil matrix in CSR
        {"name": "products_lap27_128", "kind": "products", "op": "lap27", "side": 128},
        # an unstructured matrix: uneven rows (some empty, some of hundreds
        # of entries), rectangular, as an interpolation operator or a mesh
        # of mixed elements gives
        {"name": "products_ragged_300k", "kind": "products", "op": "ragged", "rows": 300007, "cols": 290011, "mean": 18},
        # block CSR of a 3D vector problem (three unknowns a node)
        {"name": "bsr3_72", "kind": "bsr", "side": 72, "b_rows": 3, "b_cols": 3},
        # one hierarchy built from scratch: a time-dependent or nonlinear
        # problem sets up at every step
        {"name": "setup_lap27_64", "kind": "setup", "op": "lap27", "side": 64},
        # the reference's own small example: stationary V-cycles with Jacobi
        # in FP64 on 10,000 rows, bound by latency
        {"name": "solve_rot2d_100", "kind": "solve", "side": 100},
        # AMG-PCG on the headline problem: 7.08M rows, FP32 cycle
        {"name": "pcg_lap27_192_fp32", "kind": "pcg", "op": "lap27", "side": 192, "fp32": True},
        # the all-FP64 method at the middle size
        {"name": "pcg_lap27_128_fp64", "kind": "pcg", "op": "lap27", "side": 128, "fp32": False},
        # 2D anisotropic problem, many more iterations, an operator whose
        # values FP32 does not hold exactly
        {"name": "pcg_rot2d_1024_fp32", "kind": "pcg", "op": "rot2d", "side": 1024, "fp32": True},
        # several right-hand sides over one smoothed-aggregation hierarchy
        {"name": "block_sa7_96_k8", "kind": "block", "side": 96, "k": 8},
        # an uneven batch of independent 2D systems, solved together
        {"name": "batch_16", "kind": "batch", "count": 16, "lo": 64, "hi": 320, "mix": 1},
        # forward and adjoint of a variable-coefficient diffusion solve (the
        # hierarchy is built in the forward pass)
        {"name": "diff_256", "kind": "diff", "nx": 256, "ny": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["products", "products", "bsr", "setup", "solve", "pcg", "pcg", "block", "batch", "diff"])
    if kind == "products":
        op = rng.choice(["rot2d", "lap27", "ragged"])
        if op == "rot2d":
            return {"kind": kind, "op": op, "side": _log_int(rng, 40, 1200)}
        if op == "lap27":
            return {"kind": kind, "op": op, "side": _log_int(rng, 12, 128)}
        rows = _log_int(rng, 1000, 300000)
        return {"kind": kind, "op": op, "rows": rows, "cols": int(rows * rng.uniform(0.3, 1.5)) + 1, "mean": rng.randint(3, 30)}
    if kind == "bsr":
        br = rng.randint(1, 6)
        bc = br if rng.random() < 0.7 else rng.randint(1, 6)
        return {"kind": kind, "side": _log_int(rng, 10, 72 if br * bc <= 9 else 48), "b_rows": br, "b_cols": bc}
    if kind == "setup":
        op = rng.choice(["rot2d", "lap27"])
        return {"kind": kind, "op": op, "side": _log_int(rng, 64, 400) if op == "rot2d" else _log_int(rng, 16, 64)}
    if kind == "solve":
        return {"kind": kind, "side": _log_int(rng, 40, 200)}
    if kind == "pcg":
        op = rng.choice(["rot2d", "lap27"])
        fp32 = rng.random() < 0.6
        side = _log_int(rng, 64, 1024) if op == "rot2d" else _log_int(rng, 20, 192 if fp32 else 128)
        return {"kind": kind, "op": op, "side": side, "fp32": fp32}
    if kind == "block":
        return {"kind": kind, "side": _log_int(rng, 24, 96), "k": rng.choice([2, 3, 4, 5, 8])}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 16), "lo": rng.randint(32, 64), "hi": _log_int(rng, 96, 320), "mix": rng.randint(2, 10000)}
    return {"kind": kind, "nx": _log_int(rng, 48, 256), "ny": _log_int(rng, 48, 256)}


# ----------------------------------------------------------------- inputs --
# Shared by prepare() and exact(): everything here is plain torch and numpy.
def _uniform(n, seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (salt + 1) + int(seed))
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 2.0 - 1.0


def _ragged(case, seed):
    """Rows of very different lengths whose columns lie in a window around
    the (scaled) diagonal, in increasing order."""
    rng = np.random.default_rng(int(seed))
    n, m = case["rows"], case["cols"]
    lens = np.minimum(rng.pareto(2.5, n) * case["mean"] * 1.5, 40.0 * case["mean"]).astype(np.int64)
    lens[rng.random(n) < 0.02] = 0
    rows = np.repeat(np.arange(n, dtype=np.int64), lens)
    cols = rows * m // n + rng.integers(-2048, 2049, len(rows))
    cols = np.clip(cols, 0, m - 1)
    cols = cols[np.argsort(rows * m + cols, kind="stable")]
    rowptr = np.zeros(n + 1, np.int32)
    rowptr[1:] = np.cumsum(lens)
    return rowptr, cols.astype(np.int32), rng.uniform(-1.0, 1.0, len(rows))


def _bsr_arrays(case, seed):
    """Periodic 7-point pattern on a cube of nodes, uniform blocks."""
    m = case["side"]
    idx = np.arange(m ** 3).reshape(m, m, m)
    steps = [(0, 0, 0), (-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)]
    cols = np.stack([np.roll(idx, tuple(-d for d in s), axis=(0, 1, 2)).reshape(-1) for s in steps], axis=1)
    rowptr = (np.arange(m ** 3 + 1) * 7).astype(np.int32)
    vals = np.random.default_rng(int(seed)).uniform(-1.0, 1.0, (7 * m ** 3, case["b_rows"], case["b_cols"]))
    return rowptr, cols.astype(np.int32).reshape(-1), vals


def _rot2d_stencil(eps, theta):
    c, s = math.cos(theta), math.sin(theta)
    cs, cc, ss = c * s, c * c, s * s
    v1 = ((-eps - 1) * cc + (-eps - 1) * ss + (3 * eps - 3) * cs) / 6.0
    v2 = ((2 * eps - 4) * cc + (-4 * eps + 2) * ss) / 6.0
    v3 = ((-eps - 1) * cc + (-eps - 1) * ss + (-3 * eps + 3) * cs) / 6.0
    v4 = ((-4 * eps + 2) * cc + (2 * eps - 4) * ss) / 6.0
    v5 = ((8 * eps + 8) * cc + (8 * eps + 8) * ss) / 6.0
    return [v1, v2, v3, v4, v5, v4, v3, v2, v1]


def _aniso7_stencil(cz):
    st = [0.0] * 27
    st[13] = 4.0 + 2.0 * cz
    st[12] = st[14] = st[10] = st[16] = -1.0
    st[4] = st[22] = -cz
    return st


def _systems(case):
    """(side, eps, theta) of each system of a batch."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["count"]):
        side = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        out.append((side, math.exp(rng.uniform(math.log(1e-3), 0.0)), rng.uniform(0.0, math.pi)))
    return out


def _conductivity(case, seed):
    """exp of a smooth random field of about unit variance."""
    nx, ny = case["nx"], case["ny"]
    rng = np.random.default_rng(int(seed))
    y, x = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    g = np.zeros((ny, nx))
    for _ in range(24):
        kx, ky = rng.normal(0.0, 1.0 / 32.0, 2)
        g += math.sqrt(2.0 / 24) * np.cos(kx * x + ky * y + rng.uniform(0.0, 2 * math.pi))
    return torch.from_numpy(np.exp(g).reshape(-1)).cuda()


# ---------------------------------------------------------------- handles --
class _Memory:
    """Device memory of a library handle, kept alive by the tensor made of it."""

    def __init__(self, owner, ptr, n, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": kind, "data": (int(ptr), False), "version": 3}


def _view(v):
    return torch.as_tensor(_Memory(v, v.device_ptr(), v.local_n, "<f8"), device="cuda")


def _matrix_views(M):
    n, _, z = M.info()
    p = [ctypes.c_void_p() for _ in range(3)]
    rb.check(rb.lib().rb_csr_device_arrays(M.h, ctypes.byref(p[0]), ctypes.byref(p[1]), ctypes.byref(p[2])))
    return [torch.as_tensor(_Memory(M, q.value, k, t), device="cuda") for q, k, t in zip(p, (n + 1, z, z), ("<i4", "<i4", "<f8"))]


def _vector(t):
    v = rb.ParVector(t.numel())
    rb.synchronize()   # the library's stream is its own
    _view(v).copy_(t)
    return v


def _operator(case, scale=1.0):
    op, s = case["op"], case.get("side")
    if op == "lap27":
        return rb.par_stencil_grid(rb.laplace_stencil_27pt() * scale, [s, s, s])
    return rb.par_stencil_grid(rb.diffusion_stencil_2d(EPS, THETA) * scale, [s, s])


def prepare(case, seed):
    rb.init(0)
    kind, s = case["kind"], {"kind": case["kind"]}
    if kind in ("products", "bsr"):
        if kind == "bsr":
            m = case["side"] ** 3
            A = rb.BSRMatrix.from_arrays(m, m, case["b_rows"], case["b_cols"], *_bsr_arrays(case, seed))
            n, c = m * case["b_rows"], m * case["b_cols"]
        elif case["op"] == "ragged":
            n, c = case["rows"], case["cols"]
            A = rb.ParCSRMatrix.from_arrays(n, c, *_ragged(case, seed))
        else:
            A = _operator(case)
            n, c, _ = A.info()
        s.update(A=A, x=_vector(_uniform(c, seed, 1)), u=_vector(_uniform(n, seed, 2)), b=rb.ParVector(n), r=rb.ParVector(n), t=rb.ParVector(c), a0=_vector(_uniform(n, seed, 3)), a=rb.ParVector(n))
        s["out"] = [_view(s[k]) for k in ("b", "r", "t", "a")]
    elif kind == "setup":
        # the operator scaled by a power of two of the seed's (a time step's
        # factor): the same patterns, other values
        s.update(A=_operator(case, 2.0 ** (int(seed) % 31 - 15)), op=case["op"])
    elif kind == "diff":
        n = case["nx"] * case["ny"]
        s.update(k=_conductivity(case, seed).requires_grad_(True), rhs=_uniform(n, seed, 1).requires_grad_(True), target=_uniform(n, seed, 2) * 0.5 + 0.5, nx=case["nx"], ny=case["ny"])
    elif kind == "batch":
        mats = [rb.par_stencil_grid(rb.diffusion_stencil_2d(e, t), [side, side]) for side, e, t in _systems(case)]
        ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.Extended, rb.Classical, rb.L1Jacobi)
        ml.precision = rb.FP32
        B = rb.Batch(mats, ml)
        s.update(batch=B, b=_vector(_uniform(B.total_rows, seed, 1)), x=rb.ParVector(B.total_rows))
    else:
        k = case.get("k", 1)
        if kind == "block":
            m = case["side"]
            A = rb.par_stencil_grid(_aniso7_stencil(0.01), [m, m, m])
            ml = rb.ParSmoothedAggregationSolver(0.25, relax_type=rb.L1Jacobi)
            ml.precision = rb.FP32
        elif kind == "solve":
            A = _operator({"op": "rot2d", "side": case["side"]})
            ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.ModClassical, rb.Classical, rb.Jacobi)
            ml.relax_weight = 2.0 / 3.0
            ml.solve_tol = TOL
            ml.max_iterations = 2000
        else:
            A = _operator(case)
            ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.Extended, rb.Classical, rb.L1Jacobi)
            ml.precision = rb.FP32 if case["fp32"] else rb.FP64
        ml.setup(A)
        n = A.global_num_rows * k
        s.update(A=A, ml=ml, b=_vector(_uniform(n, seed, 1)), x=rb.ParVector(n), k=k)
    if "x" in s and "out" not in s:
        s["out"] = _view(s["x"])
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind in ("products", "bsr"):
        A, x, a = s["A"], s["x"], s["a"]
        a.copy(s["a0"])
        A.mult(x, s["b"])
        A.residual(x, s["u"], s["r"])
        A.mult_T(s["u"], s["t"])
        A.mult_append(x, a)
        return s["out"]
    if kind == "setup":
        if s["op"] == "lap27":
            ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.Extended, rb.Classical, rb.L1Jacobi)
            ml.precision = rb.FP32
        else:
            ml = rb.ParRugeStubenSolver(0.25, rb.PMIS, rb.ModClassical, rb.Classical, rb.Jacobi)
        ml.setup(s["A"])
        L = ml.num_levels
        return [[_matrix_views(ml.level_matrix(l, "P")) for l in range(L - 1)], [_matrix_views(ml.level_matrix(l, "A")) for l in range(1, L)]]
    if kind == "diff":
        x = rb.autograd.DiffusionSolve.apply(s["k"], s["rhs"], s["nx"], s["ny"])
        gk, gb = torch.autograd.grad(x, (s["k"], s["rhs"]), x.detach() - s["target"])
        return x.detach(), gk, gb
    s["x"].set_const_value(0.0)
    if kind == "batch":
        s["batch"].pcg(s["x"], s["b"], tol=TOL, max_iter=500)
    elif kind == "block":
        rb.PCG_block(s["A"], s["ml"], s["x"], s["b"], s["k"], tol=TOL, max_iter=500)
    elif kind == "solve":
        s["ml"].solve(s["x"], s["b"])
    else:
        rb.PCG(s["A"], s["ml"], s["x"], s["b"], [], tol=TOL, max_iter=500, mode=rb.PCG_TRUE_RESIDUAL)
    return s["out"]


# ------------------------------------------------------------------ exact --
def _product(rows, cols, vals, x, n):
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, rows, vals * x[cols])


def _stencil_entries(st, dims):
    """Rows, columns and values of a stencil on a box with zero walls."""
    shape = tuple(dims)
    idx = torch.arange(int(np.prod(shape)), device="cuda").reshape(shape)
    R, Cc, V = [], [], []
    for k, v in enumerate(st):
        if v == 0.0:
            continue
        off = [(k // 3 ** (len(shape) - 1 - d)) % 3 - 1 for d in range(len(shape))]
        here = tuple(slice(max(0, -o), m - max(0, o)) for o, m in zip(off, shape))
        there = tuple(slice(max(0, o), m + min(0, o)) for o, m in zip(off, shape))
        R.append(idx[here].reshape(-1))
        Cc.append(idx[there].reshape(-1))
        V.append(torch.full((R[-1].numel(),), v, dtype=torch.float64, device="cuda"))
    return torch.cat(R), torch.cat(Cc), torch.cat(V)


def _sines(m):
    """Eigenvectors (columns) and 2 cos(j pi / (m + 1)) of the tridiagonal
    matrix with zeros on and ones off the diagonal."""
    j = torch.arange(1, m + 1, dtype=torch.float64, device="cuda")
    Q = torch.sin(j[:, None] * j[None, :] * (math.pi / (m + 1))) * math.sqrt(2.0 / (m + 1))
    return Q, 2.0 * torch.cos(j * (math.pi / (m + 1)))


def _tensor_solve(m, eig, b):
    """x with A x = b, A diagonal (eig) in the sine basis of an m^3 cube;
    b has m^3 rows and any number of columns."""
    Q, _ = _sines(m)
    w = b.reshape(m, m, m, -1)

    def forth(v):
        v = torch.einsum("ai,ijkc->ajkc", Q, v)
        v = torch.einsum("bj,ajkc->abkc", Q, v)
        return torch.einsum("dk,abkc->abdc", Q, v)

    return forth(forth(w) / eig[..., None]).reshape(b.shape)


def _band_solve(diag, lower, upper, b):
    """Block tridiagonal solve, one dense block a grid line: diag(i),
    lower(i) (to line i - 1) and upper(i) (to line i + 1) give the blocks."""
    ny = b.shape[0]
    F, y = [], []
    for i in range(ny):
        D, r = diag(i).clone(), b[i].clone()
        if i:
            W = torch.linalg.lu_solve(*F[-1], torch.cat([upper(i - 1), y[-1][:, None]], dim=1))
            D -= lower(i) @ W[:, :-1]
            r -= lower(i) @ W[:, -1]
        F.append(torch.linalg.lu_factor(D))
        y.append(r)
    x = [None] * ny
    for i in range(ny - 1, -1, -1):
        r = y[i] if i == ny - 1 else y[i] - upper(i) @ x[i + 1]
        x[i] = torch.linalg.lu_solve(*F[i], r[:, None])[:, 0]
    return torch.stack(x)


def _tri(n, a, d, c):
    M = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    M.diagonal().fill_(d)
    if n > 1:
        M.diagonal(-1).fill_(a)
        M.diagonal(1).fill_(c)
    return M


def _rot2d_solve(side, eps, theta, b):
    v = _rot2d_stencil(eps, theta)
    lo, D, up = _tri(side, *v[0:3]), _tri(side, *v[3:6]), _tri(side, *v[6:9])
    solve = lambda r: _band_solve(lambda i: D, lambda i: lo, lambda i: up, r.reshape(side, side)).reshape(-1)  # noqa: E731
    x = solve(b)
    R, Cc, V = _stencil_entries(v, (side, side))
    return x + solve(b - _product(R, Cc, V, x, side * side))


def _diff_exact(case, seed):
    nx, ny = case["nx"], case["ny"]
    k = _conductivity(case, seed).reshape(ny, nx)
    b = _uniform(nx * ny, seed, 1).reshape(ny, nx)
    target = (_uniform(nx * ny, seed, 2) * 0.5 + 0.5).reshape(ny, nx)
    th = 2 * k[:, 1:] * k[:, :-1] / (k[:, 1:] + k[:, :-1])
    tv = 2 * k[1:] * k[:-1] / (k[1:] + k[:-1])
    d = torch.zeros_like(k)
    d[:, 1:] += th
    d[:, :-1] += th
    d[1:] += tv
    d[:-1] += tv
    d[0] += 2 * k[0]
    d[-1] += 2 * k[-1]
    d[:, 0] += 2 * k[:, 0]
    d[:, -1] += 2 * k[:, -1]

    def block(i):
        M = torch.diag(d[i])
        M.diagonal(1).copy_(-th[i])
        M.diagonal(-1).copy_(-th[i])
        return M

    link = lambda i: torch.diag(-tv[i])  # noqa: E731

    def apply(x):
        r = d * x
        r[:, 1:] -= th * x[:, :-1]
        r[:, :-1] -= th * x[:, 1:]
        r[1:] -= tv * x[:-1]
        r[:-1] -= tv * x[1:]
        return r

    def solve(f):
        x = _band_solve(block, lambda i: link(i - 1), link, f)
        return x + _band_solve(block, lambda i: link(i - 1), link, f - apply(x))

    x = solve(b)
    lam = solve(x - target)
    gk = torch.zeros_like(k)
    gh = -(lam[:, 1:] - lam[:, :-1]) * (x[:, 1:] - x[:, :-1])
    gv = -(lam[1:] - lam[:-1]) * (x[1:] - x[:-1])
    sh, sv = (k[:, 1:] + k[:, :-1]) ** 2, (k[1:] + k[:-1]) ** 2
    gk[:, :-1] += gh * 2 * k[:, 1:] ** 2 / sh
    gk[:, 1:] += gh * 2 * k[:, :-1] ** 2 / sh
    gk[:-1] += gv * 2 * k[1:] ** 2 / sv
    gk[1:] += gv * 2 * k[:-1] ** 2 / sv
    wall = -2 * lam * x
    gk[0] += wall[0]
    gk[-1] += wall[-1]
    gk[:, 0] += wall[:, 0]
    gk[:, -1] += wall[:, -1]
    return x.reshape(-1), gk.reshape(-1), lam.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "setup":
        return None   # its integers and FP64 values are compared as they are
    if kind in ("products", "bsr"):
        if kind == "bsr":
            m = case["side"] ** 3
            br, bc = case["b_rows"], case["b_cols"]
            rowptr, cols, vals = _bsr_arrays(case, seed)
            n, c = m * br, m * bc
            bi = np.repeat(np.arange(m), np.diff(rowptr))
            R = torch.from_numpy(bi).cuda()[:, None, None] * br + torch.arange(br, device="cuda")[None, :, None]
            Cc = torch.from_numpy(cols.astype(np.int64)).cuda()[:, None, None] * bc + torch.arange(bc, device="cuda")[None, None, :]
            V = torch.from_numpy(vals).cuda()
            R, Cc, V = (t.expand(V.shape).reshape(-1) for t in (R, Cc, V))
        elif case["op"] == "ragged":
            n, c = case["rows"], case["cols"]
            rowptr, cols, vals = _ragged(case, seed)
            R = torch.from_numpy(np.repeat(np.arange(n), np.diff(rowptr))).cuda()
            Cc, V = torch.from_numpy(cols.astype(np.int64)).cuda(), torch.from_numpy(vals).cuda()
        else:
            s = case["side"]
            lap = [-1.0] * 27
            lap[13] = 26.0
            R, Cc, V = _stencil_entries(lap, (s, s, s)) if case["op"] == "lap27" else _stencil_entries(_rot2d_stencil(EPS, THETA), (s, s))
            n = c = s ** (3 if case["op"] == "lap27" else 2)
        x, u, a0 = _uniform(c, seed, 1), _uniform(n, seed, 2), _uniform(n, seed, 3)
        b = _product(R, Cc, V, x, n)
        return [b, u - b, _product(Cc, R, V, u, c), a0 + b]
    if kind == "diff":
        return _diff_exact(case, seed)
    if kind == "batch":
        sides = _systems(case)
        b = _uniform(sum(m * m for m, _, _ in sides), seed, 1)
        parts = b.split([m * m for m, _, _ in sides])
        return torch.cat([_rot2d_solve(m, e, t, p) for (m, e, t), p in zip(sides, parts)])
    m = case["side"]
    if kind == "block":
        _, w = _sines(m)
        eig = (2.0 + 2.0 * 0.01 - 0.01 * w)[:, None, None] + (1.0 - w)[None, :, None] + (1.0 - w)[None, None, :]
        return _tensor_solve(m, eig, _uniform(m ** 3 * case["k"], seed, 1).reshape(m ** 3, -1)).reshape(-1)
    if kind == "pcg" and case["op"] == "lap27":
        _, w = _sines(m)
        p = 1.0 + w
        eig = 27.0 - p[:, None, None] * p[None, :, None] * p[None, None, :]
        return _tensor_solve(m, eig, _uniform(m ** 3, seed, 1).reshape(-1, 1)).reshape(-1)
    return _rot2d_solve(m, EPS, THETA, _uniform(m * m, seed, 1))


# ------------------------------------------------------------------- work --
def _entries(op, m):
    return (3 * m - 2) ** (3 if op == "lap27" else 2)


def work(case):
    """Solves: every iteration applies the operator, two sweeps, a residual
    and the vector updates on the finest grid (a constant-coefficient stencil
    needs no stored values: 12 vectors of 8 bytes a row) and the coarser
    levels' matrices, which hold about as much as the finest vectors."""
    kind = case["kind"]
    if kind == "products":
        if case["op"] == "ragged":
            n, c, z = case["rows"], case["cols"], int(case["rows"] * case["mean"])
        else:
            n = c = case["side"] ** (3 if case["op"] == "lap27" else 2)
            z = _entries(case["op"], case["side"])
        return {"bytes": 4 * (12 * z + 4 * n) + 8 * (4 * n + 3 * n + 4 * c), "flops": 8 * z}
    if kind == "bsr":
        m, e = case["side"] ** 3, case["b_rows"] * case["b_cols"]
        z = 7 * m
        return {"bytes": 4 * (z * (8 * e + 4) + 4 * m) + 8 * m * (7 * case["b_rows"] + 4 * case["b_cols"]), "flops": 8 * z * e}
    if kind == "setup":
        n, z = case["side"] ** (3 if case["op"] == "lap27" else 2), _entries(case["op"], case["side"])
        # A read, about as much again written as P, R and the coarse matrices
        return {"bytes": 2 * (12 * z + 4 * n), "flops": 20 * z}
    if kind == "diff":
        n = case["nx"] * case["ny"]
        return {"bytes": 2 * 15 * 200 * n, "flops": 2 * 15 * 100 * n}
    if kind == "batch":
        n = sum(m * m for m, _, _ in _systems(case))
        return {"bytes": 20 * 200 * n, "flops": 20 * 120 * n}
    n = case["side"] ** (3 if kind == "block" or case.get("op") == "lap27" else 2)
    its, row = {"solve": (40, 150), "block": (23, 150)}.get(kind, (13, 150) if case.get("op") == "lap27" else (40, 180))
    if kind == "block":
        return {"bytes": its * n * (60 + 90 * case["k"]), "flops": its * n * 60 * case["k"]}
    scale = 1.0 if kind == "solve" or not case["fp32"] else 0.7
    return {"bytes": its * row * scale * n, "flops": its * 200 * n}


def tolerance(case):
    """Products: FP64 sums in another order.  Solves: two correct runs stop
    at residuals below 1e-8 that need not be the same one, so their solutions
    agree to that times what the operator amplifies.  Setup: whole numbers
    and FP64 values of a fixed order of operations."""
    kind = case["kind"]
    if kind == "setup":
        return "exact"
    if kind in ("products", "bsr"):
        return {"rel": 2e-15, "max": 1e-13}
    if kind == "diff":
        return {"rel": 5e-10, "max": 5e-8}
    return {"rel": 1e-6 if kind == "solve" else 1e-7, "max": 1e-5}
