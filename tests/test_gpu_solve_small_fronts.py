"""Solve sweeps over small fronts with every kind of right-hand-side count (-m gpu):
the 8-, 16- and 32-lane groups and the five rows per lane, the passes of one, two
and eight right-hand sides, the groups of eight and a last group of one.

Oracle: the dense system's residual in FP64.  Tolerances as for the large fronts
in test_gpu_front_sizes.py: a backward stable solve leaves n eps of the norms
(n below 250), an FP32 factor's sqrt(n) u_32 cond.
"""
import numpy as np
import pytest

import mdgpu_b200 as M
from tests.test_gpu_front_sizes import SIZES, SMALL, _leaves, _two_leaves

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected only on GPU boxes
    pytest.skip("needs a CUDA device", allow_module_level=True)


@pytest.mark.parametrize("cs,u", SMALL)
@pytest.mark.parametrize("prec,tol", [(M.FP64, 1e-14), (M.FP32, 2e-5)])
def test_small_front_solves(cs, u, prec, tol):
    n, A, Ap, Ai, Ax = _leaves(cs, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    assert S.info("large_fronts") == 0
    S.factor(torch.from_numpy(Ax).cuda(), prec)
    B = np.random.default_rng(6).uniform(-1.0, 1.0, (n, 17))
    scale = np.abs(A).sum(1).max()
    for k in (1, 2, 3, 7, 8, 9, 17):
        X = S.solve(B[:, :k]).reshape(n, k)
        r = np.abs(B[:, :k] - A @ X).max(0)
        assert (r <= tol * (scale * np.abs(X).max(0) + np.abs(B[:, :k]).max(0))).all(), k


@pytest.mark.parametrize("fronts", [_leaves(*a) for a in SMALL[::3]] +
                         [_two_leaves(*a) for a in SIZES[::3]])
@pytest.mark.parametrize("prec", [M.FP64, M.FP32])
def test_columns_do_not_depend_on_the_columns_beside_them(fronts, prec):
    """Also a last group of one column (9, 17 and 57 right-hand sides).  Only a
    single right-hand side takes sums of another order."""
    n, A, Ap, Ai, Ax = fronts
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), prec)
    B = np.random.default_rng(7).uniform(-1.0, 1.0, (n, 64))
    full = S.solve(B)
    for k in (2, 3, 8, 9, 10, 17, 57):
        assert np.array_equal(S.solve(B[:, :k]), full[:, :k]), k


# leaves of one column under a root: the entries of a row of the root's front
# vector in trips of eight, four and two, a child at a time or two
@pytest.mark.parametrize("leaves", [1, 2, 3, 4, 5, 7, 8, 9, 11, 16, 35])
@pytest.mark.parametrize("u", [6, 60, 200])
@pytest.mark.parametrize("prec,tol", [(M.FP64, 1e-14), (M.FP32, 2e-5)])
def test_many_children(leaves, u, prec, tol):
    n, A, Ap, Ai, Ax = _leaves((1,) * leaves, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), prec)
    B = np.random.default_rng(9).uniform(-1.0, 1.0, (n, 10))
    scale = np.abs(A).sum(1).max()
    for k in (1, 2, 10):
        X = S.solve(B[:, :k]).reshape(n, k)
        r = np.abs(B[:, :k] - A @ X).max(0)
        assert (r <= tol * (scale * np.abs(X).max(0) + np.abs(B[:, :k]).max(0))).all(), k
