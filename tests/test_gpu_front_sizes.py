"""Fronts of chosen sizes (-m gpu): two leaf fronts of c1 and c2 pivot columns
under one root of u rows, every block dense, so each front's rows and pivot
columns sit where the kernels' tiles end (64 x 64 pieces, 128-tiles,
256-column panels, the small / large boundary at 160 rows, odd leading rows).

Oracle: dense FP64 numpy on the same matrix.  Tolerance: a backward stable
Cholesky of order n and condition k returns L to n eps k; the matrices here
are diagonally dominant with condition below 10 and n below 1000, so 1e-12
leaves a factor of ten over 1000 * 2.2e-16 * 0.5.
"""
import contextlib

import numpy as np
import pytest

import mdgpu_b200 as M

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected only on GPU boxes
    pytest.skip("needs a CUDA device", allow_module_level=True)

SIZES = [(1, 2, 161), (33, 97, 64), (64, 65, 127), (63, 129, 128), (161, 31, 130), (255, 192, 33),
         (256, 257, 191), (300, 64, 257)]


# leaves of the pivot columns given, under a root of u rows, all of them fronts
# of at most 160 rows: the edges of the 8, 16 and 32 rows of a lane group, of the
# eight-column panels, of the 32-row blocks; more children than a warp has lanes
SMALL = [((1, 2, 7), 1), ((1, 3), 6), ((4, 1), 12), ((9, 1), 7), ((1,) * 70, 15), ((17, 8, 1), 24),
         ((7, 8, 9), 23), ((1,) * 33 + (31, 32), 33), ((16, 64), 65), ((63, 1, 33), 96),
         ((24, 95, 40), 64), ((1,) * 40 + (127,), 33), ((2, 80, 60), 80), ((1, 31), 129),
         ((152,), 8), ((3, 5), 155)]


def _leaves(cs, u, seed=0):
    """Dense symmetric matrix of the pattern of the leaves, its lower CSC."""
    beg = np.concatenate([[0], np.cumsum(cs)])
    n = beg[-1] + u
    leaf = np.concatenate([np.repeat(np.arange(len(cs)), cs), np.full(u, -1)])
    r = np.random.default_rng(seed)
    A = r.uniform(-1.0, 1.0, (n, n))
    A = 0.5 * (A + A.T)
    A[(leaf[:, None] != leaf[None, :]) & (leaf[:, None] >= 0) & (leaf[None, :] >= 0)] = 0.0
    np.fill_diagonal(A, 1.5 * np.abs(A).sum(axis=1))
    Ai = [j + np.flatnonzero((leaf[j:] == leaf[j]) | (leaf[j:] < 0)) for j in range(n)]
    cols = np.repeat(np.arange(n), [len(a) for a in Ai])
    Ap = np.concatenate([[0], np.cumsum([len(a) for a in Ai])])
    Ai = np.concatenate(Ai)
    return n, A, Ap.astype(np.int32), Ai.astype(np.int32), A[Ai, cols]


def _two_leaves(c1, c2, u, seed=0):
    """Dense symmetric matrix of the two-leaf pattern and its lower CSC."""
    n = c1 + c2 + u
    r = np.random.default_rng(seed)
    A = r.uniform(-1.0, 1.0, (n, n))
    A = 0.5 * (A + A.T)
    A[c1:c1 + c2, :c1] = 0.0
    A[:c1, c1:c1 + c2] = 0.0
    np.fill_diagonal(A, 1.5 * np.abs(A).sum(axis=1))
    Ai, Ap = [], [0]
    for j in range(n):
        rows = np.arange(j, n)
        if j < c1:
            rows = rows[(rows < c1) | (rows >= c1 + c2)]
        Ai.append(rows)
        Ap.append(Ap[-1] + len(rows))
    Ai = np.concatenate(Ai)
    cols = np.repeat(np.arange(n), np.diff(Ap))
    return n, A, np.array(Ap, np.int32), Ai.astype(np.int32), A[Ai, cols]


def _dense_L(S):
    Lp, Li, Lx = S.get_L()
    L = np.zeros((S.n, S.n))
    L[Li, np.repeat(np.arange(S.n), np.diff(Lp))] = Lx
    return L


@pytest.mark.parametrize("c1,c2,u", SIZES)
def test_fp64_factor(c1, c2, u):
    n, A, Ap, Ai, Ax = _two_leaves(c1, c2, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), M.FP64)
    ref = np.linalg.cholesky(A)
    assert np.linalg.norm(_dense_L(S) - ref) <= 1e-12 * np.linalg.norm(ref)


@pytest.mark.parametrize("c1,c2,u", SIZES)
def test_fp32_factor(c1, c2, u):
    """FP32 factor: sqrt(n) u_32 cond = 30 * 6e-8 * 10 = 2e-5 bounds the
    expected forward error of L; refinement reaches 1e-14."""
    n, A, Ap, Ai, Ax = _two_leaves(c1, c2, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), M.FP32)
    ref = np.linalg.cholesky(A)
    assert np.linalg.norm(_dense_L(S) - ref) <= 2e-5 * np.linalg.norm(ref)
    b = np.random.default_rng(1).uniform(-1.0, 1.0, n)
    x, berr, _ = S.refine(b)
    r = b - A @ x
    assert np.abs(r).max() <= 1e-14 * (np.abs(A).sum(1).max() * np.abs(x).max() + np.abs(b).max())


@pytest.mark.parametrize("c1,c2,u", SIZES)
@pytest.mark.parametrize("precision", [M.FP64, M.FP32])
def test_solve_groups(c1, c2, u, precision):
    """Right-hand sides around the groups of eight of the solve; a column's
    values do not depend on the columns beside it (each group, and each column
    of a group, is a sum of its own in a fixed order)."""
    n, A, Ap, Ai, Ax = _two_leaves(c1, c2, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), precision)
    B = np.random.default_rng(2).uniform(-1.0, 1.0, (n, 65))
    tol = 1e-14 if precision == M.FP64 else 2e-5  # as the factors' bounds above
    scale = np.abs(A).sum(1).max()
    full = None
    for k in (65, 2, 7, 8, 9, 17, 64):
        X = S.solve(B[:, :k])
        r = np.abs(B[:, :k] - A @ X).max(0)
        assert (r <= tol * (scale * np.abs(X).max(0) + np.abs(B[:, :k]).max(0))).all()
        full = X if full is None else full
        same = k if k % 8 != 1 else k - 1  # a lone last column of a pass takes the one-column sweep
        assert np.array_equal(X[:, :min(same, 64)], full[:, :min(same, 64)])


@pytest.mark.parametrize("c1,c2,u", SIZES)
def test_selected_inverse(c1, c2, u):
    """The gradient of log det A on A's pattern is the inverse there (twice it
    off the diagonal); a backward stable inverse is good to n eps cond, as L."""
    n, A, Ap, Ai, Ax = _two_leaves(c1, c2, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), M.FP64)
    sign, ref = np.linalg.slogdet(A)
    assert abs(S.logdet() - ref) <= 1e-12 * abs(ref)
    S.selinv()
    cols = np.repeat(np.arange(n), np.diff(Ap))
    Z = np.linalg.inv(A)[Ai, cols] * np.where(Ai == cols, 1.0, 2.0)
    assert np.linalg.norm(S.grad_lower() - Z) <= 1e-12 * np.linalg.norm(Z)


@pytest.mark.parametrize("c1,c2,u", SIZES)
def test_reverse_mode(c1, c2, u):
    """Abar of a random Lbar against the dense adjoint of Cholesky (Murray
    2016): two more triangular solves than the inverse, so ten times its
    bound."""
    n, A, Ap, Ai, Ax = _two_leaves(c1, c2, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), M.FP64)
    Lp, Li, _ = S.get_L(values=False)
    lbar = np.random.default_rng(3).uniform(-1.0, 1.0, len(Li))
    Lbar = np.zeros((n, n))
    Lbar[Li, np.repeat(np.arange(n), np.diff(Lp))] = lbar
    L = np.linalg.cholesky(A)
    P = np.tril(L.T @ Lbar)
    P[np.diag_indices(n)] *= 0.5
    inv = np.linalg.inv(L)
    H = 0.5 * inv.T @ (P + P.T) @ inv
    cols = np.repeat(np.arange(n), np.diff(Ap))
    ref = H[Ai, cols] * np.where(Ai == cols, 1.0, 2.0)
    assert np.linalg.norm(S.adjoint(lbar) - ref) <= 1e-11 * np.linalg.norm(ref)


# tolerances as for the large fronts' factors above (n below 250 here)
@pytest.mark.parametrize("cs,u", SMALL)
@pytest.mark.parametrize("prec,tol", [(M.FP64, 1e-12), (M.FP32, 2e-5)])
def test_small_fronts(cs, u, prec, tol):
    n, A, Ap, Ai, Ax = _leaves(cs, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), prec)
    ref = np.linalg.cholesky(A)
    assert np.linalg.norm(_dense_L(S) - ref) <= tol * np.linalg.norm(ref)


# L's columns are packed on the device 8 M values at a time: above that, several
# rounds.  ||L L' v - A v|| <= (m + 1) eps || |L| |L'| |v| || for a factor with m
# terms per row sum; rows of L here hold below 1e4 terms.
@pytest.mark.parametrize("prec,eps", [(M.FP64, 2.0 ** -52), (M.FP32, 2.0 ** -23)])
def test_get_L_in_rounds(prec, eps):
    sp = pytest.importorskip("scipy.sparse")
    from mdgpu_b200 import matgen as mg
    n, Ap, Ai, Ax = mg.laplacian_3d_varcoef(36)
    S = M.Solver(n, Ap, Ai)
    S.factor(np.asarray(Ax, np.float64), prec)
    Lp, Li, Lx = S.get_L()
    assert Lp[-1] > 8 << 20
    L = sp.csc_matrix((Lx, Li, Lp), shape=(n, n))
    A = mg.lower_to_full_scipy(n, Ap, Ai, Ax).tocsr()
    p = S.array("perm")  # new -> old
    v = np.random.default_rng(3).uniform(-1.0, 1.0, n)
    r = L @ (L.T @ v) - A[p][:, p] @ v
    bound = 1e4 * eps * (abs(L) @ (abs(L).T @ abs(v)))
    assert (np.abs(r) <= bound).all()


@pytest.mark.parametrize("cs,u", SMALL)
def test_selected_inverse_of_small_fronts(cs, u):
    """As test_selected_inverse above."""
    n, A, Ap, Ai, Ax = _leaves(cs, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), M.FP64)
    S.selinv()
    cols = np.repeat(np.arange(n), np.diff(Ap))
    Z = np.linalg.inv(A)[Ai, cols] * np.where(Ai == cols, 1.0, 2.0)
    assert np.linalg.norm(S.grad_lower() - Z) <= 1e-12 * np.linalg.norm(Z)


def _volume():
    from mdgpu_b200 import matgen as mg
    return mg.laplacian_3d_varcoef(36)


@contextlib.contextmanager
def _device_filled(free_bytes):
    """Device memory taken until about free_bytes are left."""
    torch.cuda.empty_cache()
    held = []
    try:
        for step in (256 << 20, 2 << 20):
            room = torch.cuda.mem_get_info()[0] - free_bytes
            if room >= step:
                held.append(torch.empty(room // step * step, dtype=torch.uint8, device="cuda"))
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def test_get_L_leaves_the_memory_to_later_calls():
    """A first solve with several right-hand sides, on a device with room for
    little more than its storage, works after get_L as it does without."""
    n, Ap, Ai, Ax = _volume()
    S = M.Solver(n, Ap, Ai)
    dAx = torch.from_numpy(Ax).cuda()
    S.factor(dAx, M.FP64)
    B = np.random.default_rng(5).uniform(-1.0, 1.0, (n, 64))
    S.solve(B[:, :2])  # the path's kernels loaded
    need = 8 * 64 * (5 * n + S.info("solve_work_rows"))
    with _device_filled(need + (24 << 20)):
        Lx = S.get_L()[2]
        X = S.solve(B)
    assert Lx.size > 8 << 20
    x = M.Solver(n, Ap, Ai)
    x.factor(dAx, M.FP64)
    assert np.array_equal(x.solve(B), X)


@pytest.mark.parametrize("prec", [M.FP64, M.FP32])
def test_get_L_without_room_on_the_device(prec):
    """No room for the packing buffer: the same values, packed on the host."""
    n, Ap, Ai, Ax = _volume()
    dAx = torch.from_numpy(Ax).cuda()
    S, T = M.Solver(n, Ap, Ai), M.Solver(n, Ap, Ai)
    S.factor(dAx, prec)
    T.factor(dAx, prec)
    ref = S.get_L()[2]
    with _device_filled(6 << 20):
        Lx = T.get_L()[2]
    assert np.array_equal(Lx, ref)


@pytest.mark.parametrize("systems", [147, 148, 444])
def test_selected_inverse_of_many_systems(systems):
    """Systems of a leaf front of 40 pivot columns and 230 rows (three 64-row
    tiles in its step) under a root of 230 columns (the other leaf's among them;
    one, two and three tiles in its steps).  From three tiles for each of the GPU's
    148 SMs on (148 systems' leaves, 444 systems' roots throughout) a step's sums
    are not split and its tiles finish in the same launch.  Bound as in
    test_selected_inverse above."""
    n, A, Ap, Ai, _ = _two_leaves(40, 40, 190)
    cols = np.repeat(np.arange(n), np.diff(Ap))
    vals = np.random.default_rng(8).uniform(-1.0, 1.0, (systems, len(Ai)))
    vals[:, Ai == cols] = 0.0
    D = np.zeros((systems, n, n))
    D[:, Ai, cols] = D[:, cols, Ai] = vals
    D[:, range(n), range(n)] = vals[:, Ai == cols] = 1.5 * np.abs(D).sum(2)
    S = M.Solver.batch([(n, Ap, Ai)] * systems, ordering=M.ORDER_NATURAL)
    assert S.info("large_fronts") == 2 * systems
    S.factor(torch.from_numpy(vals.ravel()).cuda(), M.FP64)
    S.selinv()
    Z = np.linalg.inv(D)[:, Ai, cols] * np.where(Ai == cols, 1.0, 2.0)
    got = S.grad_lower().reshape(Z.shape)
    assert (np.linalg.norm(got - Z, axis=1) <= 1e-12 * np.linalg.norm(Z, axis=1)).all()


# more supernodes than warps (a lane each; those of more than four columns a warp
# each).  A sum of n logarithms, each within an ulp or two: (n + 2) eps times the
# sum of their sizes.
@pytest.mark.parametrize("tree", [M.TREE_NODAL, M.TREE_SUPER])
@pytest.mark.parametrize("prec", [M.FP64, M.FP32])
def test_logdet_of_many_supernodes(tree, prec):
    from mdgpu_b200 import matgen as mg
    n, Ap, Ai, Ax = mg.laplacian_2d_5pt(80)
    S = M.Solver(n, Ap, Ai, tree=tree)
    assert S.info("nsuper") > 8 * 2 * 148
    S.factor(np.asarray(Ax, np.float64), prec)
    Lp, _, Lx = S.get_L()
    logs = 2.0 * np.log(Lx[Lp[:-1]])
    assert abs(S.logdet() - logs.sum()) <= (n + 2) * 2.0 ** -52 * np.abs(logs).sum()


@pytest.mark.parametrize("c1,c2,u", SIZES)
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("where", ["leaf", "root"])
def test_reverse_mode_of_an_odd_entry(c1, c2, u, bad, where):
    """L(r, k) does not depend on A's later columns, nor, for an update row r of a
    front, on that front's other update rows, the fronts beside it or its
    ancestors: a NaN or an infinity in Lbar(r, k) leaves their gradients what they
    are with a zero in its place (bound as in test_reverse_mode)."""
    n, A, Ap, Ai, Ax = _two_leaves(c1, c2, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), M.FP64)
    Lp, Li, _ = S.get_L(values=False)
    cols = np.repeat(np.arange(n), np.diff(Lp))
    lbar = np.random.default_rng(3).uniform(-1.0, 1.0, len(Li))
    if where == "leaf":
        k, r = c1 // 2, c1 + c2 + u // 2
        kept = (cols > k) | ((Li >= c1) & (Li != r))
    else:
        k, r = c1 + c2 + u // 3, n - 1 - u // 4
        kept = cols > k
    at = np.flatnonzero((Li == r) & (cols == k))
    assert len(at) == 1
    # A's pattern is L's here: the leaves and the root are dense
    assert np.array_equal(Lp, Ap) and np.array_equal(Li, Ai)
    lbar[at] = 0.0
    ref = S.adjoint(lbar)
    lbar[at] = bad
    got = S.adjoint(lbar)
    assert not np.isfinite(got).all()
    assert np.linalg.norm(got[kept] - ref[kept]) <= 1e-11 * np.linalg.norm(ref)
    lbar[at] = 0.0
    assert np.array_equal(S.adjoint(lbar), ref)  # nothing of it stays
