"""Timed cases of the numeric path: factor, solve, refinement, differentiation.

A case names a task, a pattern and a precision.  The patterns are the ones of
the benchmark and the tests -- 2D 5-point and 3D 7-point grid Laplacians with
lognormal edge conductances, the 27-point grid with three unknowns per node,
and batches of independent grid systems -- at sizes from a few hundred
unknowns to the 64^3 grid.  The symbolic analysis (one `Solver` per pattern)
belongs to the state: a program analyses once and factors many value sets.

Tasks:
  drop_in    host values in, L (compressed columns) and x out: what a caller
             of the plain C factor-and-solve contract asks for
  direct     factor on the device in FP64, solve
  refined    reduced-precision factor, FP64 iterative refinement to 1e-14
  gmres      reduced-precision factor, GMRES-based refinement to 1e-14
  resolve    solve with an FP64 factor kept from earlier (time stepping)
  reresolve  refinement with an FP32 factor kept from earlier
  gradient   log det A + b' A^-1 b and its gradients through torch.autograd
  reverse    factor, then a gradient on L's values carried back to A's values
"""
import numpy as np
import torch

import mdgpu_b200 as M
from mdgpu_b200 import matgen as mg
from mdgpu_b200.autograd import logdet_quad

PRECISION = {"fp64": M.FP64, "fp32": M.FP32, "bf16": M.BF16, "tf32": M.TF32}
#: independent systems of a batch: grid sides of its 2D and 3D halves
BATCH_2D, BATCH_3D = (16, 96), (8, 32)


def listed():
    return [
        # one small system, solved at once: launches and latency are all there is
        dict(name="small_2d", task="direct", grid="2d", nx=24, ny=23, nz=1, order="amd",
             precision="fp64", nrhs=1),
        # the 100 x 100 grid through the host contract: factor, L back, solve; the caller
        # brings an ordering of its own
        dict(name="drop_in_2d", task="drop_in", grid="2d", nx=100, ny=100, nz=1,
             order="dissection", precision="fp64", nrhs=1),
        # a large planar problem, odd sides, a few right-hand sides
        dict(name="plane_refined", task="refined", grid="2d", nx=333, ny=257, nz=1, order="amd",
             precision="fp32", nrhs=3),
        # the plain FP64 mode on a volume problem
        dict(name="volume_fp64", task="direct", grid="3d", nx=48, ny=48, nz=48, order="amd",
             precision="fp64", nrhs=1),
        # the benchmark's own step: 64^3, FP32 factor, refined solve
        dict(name="volume_refined", task="refined", grid="3d", nx=64, ny=64, nz=64, order="amd",
             precision="fp32", nrhs=1),
        # a time step: a new right-hand side for a factor already there
        dict(name="time_step", task="resolve", grid="3d", nx=41, ny=43, nz=45, order="amd",
             precision="fp64", nrhs=1),
        # many load cases for one factor
        dict(name="many_loads", task="reresolve", grid="3d", nx=48, ny=48, nz=48, order="amd",
             precision="fp32", nrhs=64),
        # three unknowns per node, the BF16 factor as a preconditioner
        dict(name="elastic_bf16", task="gmres", grid="elastic", nx=24, ny=24, nz=24,
             order="amd", precision="bf16", nrhs=1),
        # three unknowns per node, FP32 factor with plain refinement
        dict(name="elastic_refined", task="refined", grid="elastic", nx=32, ny=32, nz=32,
             order="amd", precision="fp32", nrhs=1),
        # independent uneven systems under one handle, four right-hand sides each
        dict(name="batch", task="refined", grid="batch", nx=96, ny=0, nz=0, order="amd",
             precision="fp32", nrhs=4),
        # a training step on the conductances of a grid
        dict(name="gradient", task="gradient", grid="3d", nx=32, ny=32, nz=32, order="amd",
             precision="fp64", nrhs=1),
        # reverse mode of the factorization itself
        dict(name="reverse", task="reverse", grid="3d", nx=19, ny=20, nz=21,
             order="dissection", precision="fp64", nrhs=1),
    ]


def _between(rng, lo, hi):
    """An integer of [lo, hi], even over its logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    task = rng.choice(["drop_in", "direct", "direct", "refined", "refined", "refined", "gmres",
                       "resolve", "reresolve", "gradient", "reverse"])
    c = dict(task=task, order="amd", precision="fp64", nrhs=1)
    grid = {"drop_in": "2d", "gradient": "3d", "reverse": "3d"}.get(task)
    if grid is None:
        grid = rng.choice(["2d", "3d", "3d", "elastic"] + ["batch"] * (task == "refined"))
    if grid == "2d":
        top = 100 if task == "drop_in" else 320
        side = [_between(rng, 16, top), _between(rng, 16, top), 1]
    elif grid == "batch":
        side = [_between(rng, 8, 96), 0, 0]
    else:
        top = {"gradient": 32, "reverse": 20, "direct": 48}.get(task, 60)
        if grid == "elastic":
            top = 24 if task == "direct" else 31
        mid = _between(rng, 8, top)
        side = [max(5, min(top, mid + rng.randint(-3, 3))) for _ in range(3)]
        if grid == "elastic":
            side = [side[0]] * 3
    c.update(grid=grid, nx=side[0], ny=side[1], nz=side[2])
    if task in ("refined", "reresolve"):
        c["precision"] = "fp32"
    if task == "gmres":
        c["precision"] = "fp32" if grid == "2d" else rng.choice(["bf16", "tf32", "fp32"])
    if task in ("drop_in", "reverse"):
        c["order"] = "dissection"
    if task in ("direct", "refined", "resolve", "reresolve"):
        c["nrhs"] = _between(rng, 1, 64) if "resolve" in task else rng.choice([1, 1, 1, 2, 4, 7])
    c["seed_sizes"] = rng.randint(0, 9999) if grid == "batch" else 0
    return c


# ---- patterns and values -------------------------------------------------

def _dissection(nx, ny, nz):
    """Geometric nested dissection of a grid, new -> old: halves first, the
    plane between them last."""
    idx = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    out = []

    def cut(a):
        if a.size <= 16:
            out.append(a.ravel())
            return
        ax = int(np.argmax(a.shape))
        k = a.shape[ax] // 2
        cut(np.take(a, range(k), ax))
        cut(np.take(a, range(k + 1, a.shape[ax]), ax))
        out.append(np.take(a, k, ax).ravel())

    cut(idx)
    return np.concatenate(out)


def _systems(case, seed):
    """[(n, Ap, Ai, Ax)] of the case's systems, values from the seed; a
    pattern depends on the case alone."""
    if case["grid"] == "batch":
        sizes = np.random.default_rng(case.get("seed_sizes", 0))
        got = []
        for k in range(case["nx"]):
            lo, hi = BATCH_2D if k % 2 == 0 else BATCH_3D
            dims = (int(sizes.integers(lo, hi + 1)),) * (2 if k % 2 == 0 else 3)
            got.append(mg.laplacian_grid(dims, seed=[seed, k], sigma=0.5, shift=1e-2))
        return got
    if case["grid"] == "elastic":
        return [mg.elasticity_3dof(case["nx"], seed=seed)]
    dims = (case["nx"], case["ny"]) + ((case["nz"],) if case["grid"] == "3d" else ())
    a = mg.laplacian_grid(dims, seed=seed, sigma=1.0,
                          shift=1e-2 if case["task"] == "gradient" else 1e-3)
    if case["order"] == "dissection":
        a = mg.permute_lower(*a, _dissection(case["nx"], case["ny"], case["nz"]))
    return [a]


def _system(case, seed):
    """The systems as one: (n, Ap, Ai, Ax), block-diagonal for a batch."""
    many = _systems(case, seed)
    if len(many) == 1:
        return many[0]
    rows = np.concatenate([[0], np.cumsum([s[0] for s in many])])
    vals = np.concatenate([[0], np.cumsum([s[1][-1] for s in many])])
    return (int(rows[-1]),
            np.concatenate([[0]] + [s[1][1:] + v for s, v in zip(many, vals)]).astype(np.int32),
            np.concatenate([s[2] + r for s, r in zip(many, rows)]).astype(np.int32),
            np.concatenate([s[3] for s in many]))


def _ordering(case):
    return M.ORDER_AMD if case["order"] == "amd" else M.ORDER_NATURAL


def _rhs(case, n, seed):
    return np.random.default_rng([seed, 1]).uniform(-1.0, 1.0, size=(case["nrhs"], n))


def _lbar(n, seed):
    """The gradient on L in column j is the row of weights w[j] times v[i]."""
    r = np.random.default_rng([seed, 2])
    return r.uniform(-1.0, 1.0, n), r.uniform(-1.0, 1.0, n)


# ---- state and pass --------------------------------------------------------

def prepare(case, seed):
    many = _systems(case, seed)
    if len(many) == 1:
        n, Ap, Ai, Ax = many[0]
        S = M.Solver(n, Ap, Ai, ordering=_ordering(case))
    else:
        S = M.Solver.batch([s[:3] for s in many], ordering=_ordering(case))
        n, Ax = S.n, np.concatenate([s[3] for s in many])
    st = {"task": case["task"], "S": S, "precision": PRECISION[case["precision"]]}
    B = _rhs(case, n, seed)
    if case["task"] == "drop_in":
        st.update(Ax=Ax, b=B[0])
        return st
    st["Ax"] = torch.from_numpy(Ax).cuda()
    st["B"] = torch.from_numpy(B).cuda().t()  # column-major (n, nrhs)
    st["X"] = torch.empty_like(st["B"].t()).t()
    if case["task"] in ("resolve", "reresolve"):
        S.factor(st["Ax"], st["precision"])
    elif case["task"] == "gradient":
        st["Ax"].requires_grad_(True)
        st["b"] = st["B"][:, 0].contiguous().requires_grad_(True)
    elif case["task"] == "reverse":
        Lp, Li, _ = S.get_L(values=False)
        w, v = _lbar(n, seed)
        st["Lbar"] = torch.from_numpy(np.repeat(w, np.diff(Lp)) * v[Li]).cuda()
    return st


def run(state):
    S, task = state["S"], state["task"]
    if task == "drop_in":
        S.factor(state["Ax"], state["precision"])
        Lp, Li, Lx = S.get_L()
        return {"Lp": Lp, "Li": Li, "Lx": Lx, "x": S.solve(state["b"])}
    if task == "direct":
        S.factor(state["Ax"], state["precision"])
        return {"x": S.solve(state["B"])}
    if task == "resolve":
        return {"x": S.solve(state["B"])}
    if task in ("refined", "reresolve"):
        if task == "refined":
            S.factor(state["Ax"], state["precision"])
        S.refine_device(state["B"], state["X"])
        return {"x": state["X"]}
    if task == "gmres":
        S.factor(state["Ax"], state["precision"])
        S.gmres_ir_device(state["B"], state["X"])
        return {"x": state["X"]}
    if task == "gradient":
        loss = logdet_quad(S, state["Ax"], state["b"])
        gA, gb = torch.autograd.grad(loss, (state["Ax"], state["b"]))
        return {"loss": loss.detach(), "grad_A": gA, "grad_b": gb}
    S.factor(state["Ax"], state["precision"])
    return {"Abar": S.adjoint(state["Lbar"])}


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    """Flops: the factor's sum of squared column counts, four per entry of L
    and right-hand side of a solve.  Bytes: A's values once, L written once by
    a factor and read once by each triangular sweep, right-hand sides and
    solutions once.  Refinement counts one correction; the gradients read L
    once and take twice the factor's flops."""
    many = _systems(case, 0)
    flops, lnz = M.estimate_batch([s[:3] for s in many], ordering=_ordering(case))
    f, lnz = float(flops.sum()), float(lnz.sum())
    n, nnz = float(sum(s[0] for s in many)), float(sum(s[1][-1] for s in many))
    size = 8.0 if case["precision"] == "fp64" else 4.0
    task, k = case["task"], case["nrhs"]
    flop, byte = 0.0, 0.0
    if task not in ("resolve", "reresolve"):
        flop, byte = f, 8.0 * nnz + size * lnz
    solves = {"refined": 2, "reresolve": 2, "gmres": 2, "reverse": 0}.get(task, 1)
    flop += solves * 4.0 * lnz * k
    byte += solves * 2.0 * size * lnz + 16.0 * n * k
    if solves == 2:  # the residual
        flop, byte = flop + 4.0 * nnz * k, byte + 12.0 * nnz
    if task == "drop_in":
        byte += 12.0 * lnz
    if task in ("gradient", "reverse"):
        flop += 2.0 * f
        byte += 8.0 * (lnz + nnz) + (8.0 * lnz if task == "reverse" else 0.0)
    return {"bytes": byte, "flops": flop}


# ---- 64-bit values by plain numpy and torch ----------------------------------

def _full(n, Ap, Ai, Ax):
    """(rows, cols, values) of the whole symmetric matrix, on the GPU."""
    c = np.repeat(np.arange(n, dtype=np.int64), np.diff(Ap))
    r = Ai.astype(np.int64)
    off = r != c
    at = [np.concatenate([r, c[off]]), np.concatenate([c, r[off]]), np.concatenate([Ax, Ax[off]])]
    return [torch.from_numpy(x).cuda() for x in at]


def _conjugate_gradients(n, Ap, Ai, Ax, B):
    """A^-1 B (n, k): Jacobi-preconditioned conjugate gradients in 64 bits,
    restarted on the true residual."""
    r, c, v = _full(n, Ap, Ai, Ax)
    A = torch.sparse_coo_tensor(torch.stack([r, c]), v, (n, n)).coalesce().to_sparse_csr()
    inv = torch.zeros(n, dtype=torch.float64, device="cuda")
    inv[r[r == c]] = 1.0 / v[r == c]
    inv = inv[:, None]
    B = torch.from_numpy(B).cuda()
    X = torch.zeros_like(B)
    for _ in range(4):
        R = B - A @ X
        Z = inv * R
        P, rz = Z.clone(), (R * Z).sum(0)
        start, D = rz.clone(), torch.zeros_like(B)
        for it in range(20000):
            Q = A @ P
            a = rz / (P * Q).sum(0).clamp_min(1e-300)
            D += a * P
            R -= a * Q
            Z = inv * R
            new = (R * Z).sum(0)
            P = Z + (new / rz.clamp_min(1e-300)) * P
            rz = new
            if it % 50 == 49 and bool((rz <= 1e-22 * start).all()):
                break
        X += D
    return X


def _dense(n, Ap, Ai, Ax):
    r, c, v = _full(n, Ap, Ai, Ax)
    D = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    D[r, c] = v
    return D


def _pattern(n, Ap, Ai):
    """L's pattern by columns (parents take their children's rows)."""
    kids, cols = [[] for _ in range(n)], []
    for j in range(n):
        s = np.unique(np.concatenate([Ai[Ap[j]:Ap[j + 1]]] + [cols[k][1:] for k in kids[j]]))
        cols.append(s)
        if s.size > 1:
            kids[s[1]].append(j)
    return (np.concatenate(cols).astype(np.int64),
            np.repeat(np.arange(n), [s.size for s in cols]))


def exact(case, seed):
    n, Ap, Ai, Ax = _system(case, seed)
    B = _rhs(case, n, seed)
    task = case["task"]
    if task in ("direct", "resolve", "refined", "reresolve", "gmres"):
        return {"x": _conjugate_gradients(n, Ap, Ai, Ax, np.ascontiguousarray(B.T))}
    cols = np.repeat(np.arange(n), np.diff(Ap))
    if task == "drop_in":
        L = torch.linalg.cholesky(_dense(n, Ap, Ai, Ax))
        r, c = _pattern(n, Ap, Ai)
        x = torch.cholesky_solve(torch.from_numpy(B[0][:, None]).cuda(), L)[:, 0]
        return {"Lp": None, "Li": None, "x": x.cpu().numpy(),
                "Lx": L[torch.from_numpy(r).cuda(), torch.from_numpy(c).cuda()].cpu().numpy()}
    at = torch.from_numpy(Ai.astype(np.int64)).cuda(), torch.from_numpy(cols).cuda()
    twice = torch.where(at[0] == at[1], 1.0, 2.0).double()
    if task == "gradient":
        L = torch.linalg.cholesky(_dense(n, Ap, Ai, Ax))
        b = torch.from_numpy(B[0]).cuda()
        x = torch.cholesky_solve(b[:, None], L)[:, 0]
        loss = 2.0 * torch.log(torch.diagonal(L)).sum() + torch.dot(b, x)
        Z = torch.cholesky_inverse(L)
        return {"loss": loss, "grad_A": twice * (Z[at] - x[at[0]] * x[at[1]]), "grad_b": 2.0 * x}
    # reverse: the adjoint of L = chol(A), P = the lower half of L' Lbar with its diagonal
    # halved, then L^-T (P + P') L^-1 halved is the symmetric gradient
    L = torch.linalg.cholesky(_dense(n, Ap, Ai, Ax))
    r, c = (torch.from_numpy(x).cuda() for x in _pattern(n, Ap, Ai))
    w, v = (torch.from_numpy(x).cuda() for x in _lbar(n, seed))
    Lbar = torch.zeros_like(L)
    Lbar[r, c] = w[c] * v[r]
    P = torch.tril(L.t() @ Lbar)
    P.diagonal().mul_(0.5)
    H = torch.linalg.solve_triangular(L.t(), P + P.t(), upper=True)
    H = 0.5 * torch.linalg.solve_triangular(L.t(), H.t().contiguous(), upper=True)
    return {"Abar": twice * H[at]}
