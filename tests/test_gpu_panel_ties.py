"""The FP64 LU's leaf on inputs full of equal magnitudes, at the edges of its row ranges.

A Sylvester Hadamard matrix with shuffled rows and random row and column signs has entries +-1 and
eliminates exactly in binary floating point (every multiplier and Schur element is a dyadic rational
of a few bits), so nearly every pivot is a tie that the first-maximum rule decides and the factors and
pivots must equal the oracle's bit for bit, however the updates are grouped.  The orders around 128 t,
256, 512, 1024 and 2048 rows are where the leaf changes its rows per thread or its number of CTAs; a
leading block of such a matrix is used for the orders that are not powers of two."""
import numpy as np
import pytest

import oracle
from mrmath_b200 import linalg as L

pytestmark = pytest.mark.gpu


def signed_hadamard(n, seed):
    h = np.ones((1, 1))
    while h.shape[0] < n:
        h = np.block([[h, h], [h, -h]])
    r = np.random.RandomState(seed)
    m = h.shape[0]
    h = h[r.permutation(m)] * r.choice([-1.0, 1.0], (m, 1)) * r.choice([-1.0, 1.0], (1, m))
    return np.ascontiguousarray(h)


@pytest.mark.parametrize("n", [32, 128, 256, 512, 1024, 2048])
def test_tied_pivots_are_the_first_maxima(ctx, n):
    a = signed_hadamard(n, n)
    ref, got = a.copy(), a.copy()
    rc, idx = oracle.lu_decomp_inplace(ref)
    st, piv = L.MatrixLUDecompInPlace(got, ctx=ctx)
    assert rc == st == 0
    assert np.array_equal(piv, idx)
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("n", [1, 7, 31, 33, 129, 255, 257, 511, 513, 1025, 2049])
def test_pivots_at_the_row_range_edges(ctx, n):
    a = np.random.RandomState(n).random_sample((n, n))
    ref, got = a.copy(), a.copy()
    rc, idx = oracle.lu_decomp_inplace(ref)
    st, piv = L.MatrixLUDecompInPlace(got, ctx=ctx)
    assert rc == st == 0
    assert np.array_equal(piv, idx)
    assert np.linalg.norm(got - ref) <= max(1e-12, n * 2.0 ** -53) * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [100, 700])
def test_infinite_and_nan_candidates(ctx, n):
    """A NaN never wins the pivot search and an infinity always does, in the first column of a leaf."""
    a = np.random.RandomState(n).random_sample((n, n))
    a[5, 0] = np.nan
    a[n - 3, 0] = -np.inf
    a[n - 2, 0] = np.inf
    ref, got = a.copy(), a.copy()
    _, idx = oracle.lu_decomp_inplace(ref)
    _, piv = L.MatrixLUDecompInPlace(got, ctx=ctx)
    assert piv[0] == idx[0] == n - 3
