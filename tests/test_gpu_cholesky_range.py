"""Cholesky at the edges of its leaf's fast path: scales where the root's iteration is replaced by sqrt
and division, zero, infinite and NaN diagonals, and orders around the leaf, CTA and panel widths."""
import numpy as np
import pytest

import oracle
from mrmath_b200 import linalg as L

pytestmark = pytest.mark.gpu


def spd(n, seed):
    g = np.random.RandomState(seed).random_sample((n, n)) - 0.5
    return g @ g.T + 0.25 * n * np.eye(n)


@pytest.mark.parametrize("n", [1, 32, 63, 65, 95, 97, 129, 257, 320])
@pytest.mark.parametrize("scale", [1e-290, 1e-249, 1.0, 1e251, 1e300])
def test_scales(ctx, n, scale):
    a = spd(n, n) * scale
    ref, got = a.copy(), a.copy()
    assert oracle.cholesky_inplace4(ref) == 0
    assert L.MatrixCholeskyInPlace4(got, ctx=ctx) == 0
    lo, lr = np.tril(got), np.tril(ref)
    assert np.linalg.norm(lo - lr) <= 1e-12 * np.linalg.norm(lr)
    assert np.array_equal(np.triu(got, 1), np.triu(a, 1))


@pytest.mark.parametrize("n,at", [(1, 0), (40, 0), (40, 31), (40, 32), (300, 255), (300, 256), (300, 299)])
@pytest.mark.parametrize("value", [0.0, -1.0, np.nan, np.inf, -np.inf])
def test_diagonals(ctx, n, at, value):
    a = spd(n, n)
    a[at, at] = value
    ref, got = a.copy(), a.copy()
    assert L.MatrixCholeskyInPlace4(got, ctx=ctx) == oracle.cholesky_inplace4(ref)
    lo, lr = np.tril(got), np.tril(ref)
    if value == np.inf:
        assert np.array_equal(np.isfinite(lo), np.isfinite(lr))
        fin = np.isfinite(lr)
        assert np.allclose(lo[fin], lr[fin], rtol=1e-10, atol=1e-12)
