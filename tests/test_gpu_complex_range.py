"""Complex LU, solve and inverse over the orders where their kernels change: one thread block or a cluster for a
leaf, one or two rows a thread, the strips' edges, blocks joined by products; ties, scales, singular systems."""
import numpy as np
import pytest

from mrmath_b200 import inputs, linalg as L

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _rand(r, n, k):
    return (2.0 * r.random_sample((n, k)) - 1.0) + 1j * (2.0 * r.random_sample((n, k)) - 1.0)


def _factor_error(a, lu, idx):
    n = a.shape[0]
    pa = a.copy()
    for i, q in enumerate(idx):
        if q != i:
            pa[[i, q]] = pa[[q, i]]
    lo, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    return np.abs(lo @ up - pa).max() / (np.abs(lo) @ np.abs(up)).max()


def _pivots(a):
    """the reference's interchanges, column by column (largest |re| + |im|, the first among equals)"""
    a, n, idx = a.copy(), a.shape[0], []
    for j in range(n):
        c = np.abs(a[j:, j].real) + np.abs(a[j:, j].imag)
        p = j + int(np.argmax(c))
        idx.append(p)
        a[[j, p]] = a[[p, j]]
        a[j + 1:, j] /= a[j, j]
        a[j + 1:, j + 1:] -= np.outer(a[j + 1:, j], a[j, j + 1:])
    return idx


# |L U - P A| <= n u |L| |U| entrywise for real arithmetic; complex products and CInv cost a small factor more
@pytest.mark.parametrize("n,k", [(1, 1), (7, 9), (31, 8), (33, 1), (64, 7), (95, 17), (128, 2), (129, 3), (160, 1), (255, 1),
                                 (257, 16), (385, 2), (1023, 2), (1025, 3), (1057, 1), (1100, 300), (2100, 1)])
def test_orders(ctx, n, k):
    r = inputs.rng(700 + n)
    a, b = _rand(r, n, n), _rand(r, n, k)
    lu = a.copy()
    st, idx = L.CplxMatrixLUDecompInPlace(lu, ctx=ctx)
    assert st == 0
    assert _factor_error(a, lu, idx) <= 8 * n * U
    if n <= 400:
        assert list(idx) == _pivots(a)
    st, x = L.CplxMatrixLinEQSolve(a, b, ctx=ctx)
    assert st == 0
    growth = max(1.0, np.abs(np.triu(lu)).max() / np.abs(a).max())
    scale = np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0)
    assert (np.abs(a @ x - b).max(axis=0) / scale).max() <= 8 * n * U * growth
    if n in (33, 257):
        inv = a.copy()
        assert L.CplxMatrixInverseInPlace(inv, ctx=ctx) == 0
        res = np.abs(a @ inv - np.eye(n)).max()
        assert res <= 8 * n * U * growth * np.abs(a).sum(axis=1).max() * np.abs(inv).max()


def _hadamard(n):
    h = np.ones((1, 1))
    while h.shape[0] < n:
        h = np.block([[h, h], [h, -h]])
    return h


@pytest.mark.parametrize("n", [32, 128, 256, 512])
def test_ties(ctx, n):
    r = inputs.rng(n)
    rows, cols = r.permutation(n), r.permutation(n)
    unit = np.array([1, 1j, -1, -1j])[r.randint(0, 4, n)][:, None]
    # rows of a Hadamard matrix in any order: every multiplier is 0 or a unit, so all arithmetic is exact, every
    # search is a tie and the first among equals is the only right answer
    a = _hadamard(n)[rows] * unit
    st, idx = L.CplxMatrixLUDecompInPlace(a.copy(), ctx=ctx)
    assert st == 0 and list(idx) == _pivots(a)
    # with its columns shuffled too, multipliers such as 1/3 occur and rounding decides between equals: a pivot
    # is one of the largest to within the rounding of the elimination before it
    a = _hadamard(n)[rows][:, cols] * unit
    lu = a.copy()
    st, idx = L.CplxMatrixLUDecompInPlace(lu, ctx=ctx)
    assert st == 0 and _factor_error(a, lu, idx) <= 8 * n * U
    low = np.tril(lu, -1)
    assert (np.abs(low.real) + np.abs(low.imag)).max() <= 2.0 ** 0.5 * (1 + 8 * n * U * np.abs(np.triu(lu)).max())


@pytest.mark.parametrize("n", [40, 200])
def test_scales_and_singular(ctx, n):
    r = inputs.rng(n + 1)
    a, b = _rand(r, n, n) + n * np.eye(n), _rand(r, n, 2)
    for e in (1000, -1000):  # outside the range of the reciprocal's correction: divisions
        st, x = L.CplxMatrixLinEQSolve(a * 2.0 ** e, b * 2.0 ** e, ctx=ctx)
        assert st == 0
        scale = np.abs(a).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max()
        assert np.abs(a @ x - b).max() / scale <= 8 * n * U
    for bad in (0.0, np.nan):
        c = _rand(r, n, n)
        c[:, n // 2] = bad
        st, _ = L.CplxMatrixLUDecompInPlace(c, ctx=ctx)
        assert st == 1
