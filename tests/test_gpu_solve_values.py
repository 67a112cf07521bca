"""Special values through the solve of the small fronts (-m gpu): what a
substitution column by column on L's pattern gives, which multiplies by no entry
that L does not have.

Fronts of at most 160 rows only: a large front applies the stored inverses of
whole tiles, zeros above the diagonal included, so an infinity there spreads
over its tile as a NaN.
"""
import numpy as np
import pytest

import mdgpu_b200 as M
from tests.test_gpu_front_sizes import SMALL, _leaves

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected only on GPU boxes
    pytest.skip("needs a CUDA device", allow_module_level=True)


def _substitute(Lp, Li, Lx, b):
    """x of L L' x = b, column by column."""
    x = b.copy()
    with np.errstate(invalid="ignore"):
        for j in range(len(b)):
            x[j] = x[j] / Lx[Lp[j]]
            r = slice(Lp[j] + 1, Lp[j + 1])
            x[Li[r]] -= Lx[r] * x[j]
        for j in reversed(range(len(b))):
            r = slice(Lp[j] + 1, Lp[j + 1])
            x[j] = (x[j] - Lx[r] @ x[Li[r]]) / Lx[Lp[j]]
    return x


# One infinite entry of the right-hand side: every term of a row's sum is then
# finite or infinite by its factors alone, so which of finite, +inf, -inf and NaN
# a row of x is does not depend on the order of the sums.  Finite rows (they share
# no path with the infinite one): n eps cond with n below 250 and a condition
# below 10, as for the factors.
@pytest.mark.parametrize("cs,u", SMALL)
@pytest.mark.parametrize("prec", [M.FP64, M.FP32])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_infinite_right_hand_side(cs, u, prec, nrhs):
    n, A, Ap, Ai, Ax = _leaves(cs, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), prec)
    Lp, Li, Lx = S.get_L()
    B = np.random.default_rng(4).uniform(-1.0, 1.0, (n, nrhs))
    clean = S.solve(B).reshape(n, nrhs)
    for at in sorted({0, cs[0] - 1, cs[0] + 1, n - u, n - 1}):
        C = np.asfortranarray(B)
        C[at, 0] = np.inf
        x = S.solve(C).reshape(n, nrhs)
        ref = _substitute(Lp, Li, Lx, C[:, 0])
        fin = np.isfinite(ref)
        np.testing.assert_array_equal(x[~fin, 0], ref[~fin])
        assert np.abs(x[fin, 0] - ref[fin]).max(initial=0.0) <= 1e-12
        assert np.array_equal(x[:, 1:], clean[:, 1:])  # the other columns are untouched


# A zero right-hand side: every product and sum is a zero, and a difference of
# zeros of the same sign is +0, so the solution is +0 throughout.
@pytest.mark.parametrize("cs,u", SMALL)
@pytest.mark.parametrize("nrhs", [1, 3])
def test_zero_right_hand_side(cs, u, nrhs):
    n, A, Ap, Ai, Ax = _leaves(cs, u)
    S = M.Solver(n, Ap, Ai, ordering=M.ORDER_NATURAL)
    S.factor(torch.from_numpy(Ax).cuda(), M.FP64)
    x = S.solve(np.zeros((n, nrhs), order="F"))
    assert not x.any() and not np.signbit(x).any()
