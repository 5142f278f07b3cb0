"""A right-hand side's solution has the same bits whatever stands in the columns beside it: infinities and NaN in some
columns send those, and only those, through the divisions.  (With right-hand sides of 2^-1018 the residual that
corrects a quotient is subnormal, and about 4 % of the quotients differ from the division's in the last place.)"""
import numpy as np
import pytest

from mrmath_b200 import inputs, linalg as L

pytestmark = pytest.mark.gpu

BAD = [np.inf, -np.inf, np.nan, 1e308]


def _spoil(b, r):
    """some columns with an entry that makes their solution not finite (or nearly so); the others' indexes"""
    b = b.copy()
    cols = r.permutation(b.shape[1])[: max(1, b.shape[1] // 3)]
    for c in cols:
        b[r.randint(b.shape[0]), c] = BAD[r.randint(len(BAD))]
    return b, np.setdiff1d(np.arange(b.shape[1]), cols)


@pytest.mark.parametrize("n,k", [(5, 2), (32, 8), (100, 3), (256, 70), (300, 5), (300, 80), (520, 1200)])
@pytest.mark.parametrize("e", [0, -1018])
def test_solve(ctx, n, k, e):
    import torch
    r = inputs.rng(n + k)
    a, b = 2.0 * r.random_sample((n, n)) - 1.0, np.ldexp(r.standard_normal((n, k)), e)
    bad, rest = _spoil(b, r)
    out = []
    for rhs in (b, bad):
        X = torch.empty((n, k), dtype=torch.float64, device="cuda")
        L.dev_MatrixLinEQSolve(torch.from_numpy(a).cuda(), torch.from_numpy(rhs).cuda(), X, ctx=ctx)
        out.append(X.cpu().numpy())
    assert np.array_equal(out[0][:, rest], out[1][:, rest])


@pytest.mark.parametrize("n,k", [(7, 2), (40, 9), (600, 12)])
@pytest.mark.parametrize("e", [0, -1018])
def test_complex_solve(ctx, n, k, e):
    r = inputs.rng(n + k)
    a = (r.random_sample((n, n)) - 0.5) + 1j * (r.random_sample((n, n)) - 0.5)
    b = np.ldexp(r.standard_normal((n, k)), e) + 1j * np.ldexp(r.standard_normal((n, k)), e)
    bad, rest = _spoil(b, r)
    x, y = L.CplxMatrixLinEQSolve(a, b, ctx=ctx)[1], L.CplxMatrixLinEQSolve(a, bad, ctx=ctx)[1]
    assert np.array_equal(x[:, rest], y[:, rest])


@pytest.mark.parametrize("e", [0, -1018])
def test_batch(ctx, e):
    r = inputs.rng(3)
    mats = [2.0 * r.random_sample((n, n)) - 1.0 + n * np.eye(n) for n in (8, 33, 64, 100, 128, 200, 256) * 3]
    rhss = [np.ldexp(r.standard_normal((m.shape[0], 8)), e) for m in mats]
    bad, rest = zip(*(_spoil(b, r) for b in rhss))
    x, y = L.BatchLinEQSolve(mats, rhss, ctx=ctx)[0], L.BatchLinEQSolve(mats, list(bad), ctx=ctx)[0]
    for p, q, c in zip(x, y, rest):
        assert np.array_equal(p[:, c], q[:, c])
