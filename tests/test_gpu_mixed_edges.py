"""The mixed solve's pivot tournament at its edges: leaves narrower than a block of eight columns and up to 32,
last chunks of a few rows (fewer than the leaf is wide), rows that tie, columns that vanish in one chunk only."""
import numpy as np
import pytest

import oracle
from mrmath_b200 import _lib, inputs, linalg as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 17, 31, 33, 40, 65, 511, 512, 513, 519, 543, 545, 1025, 1056])
def test_edge_orders(ctx, n):
    r = inputs.rng(60 + n)
    a, b = 2.0 * r.random_sample((n, n)) - 1.0, r.standard_normal((n, 2))
    a += 0.5 * np.sqrt(n) * np.eye(n)[r.permutation(n)]  # (well conditioned: the FP32 factors refine)
    st, x, rep = L.MatrixLinEQSolveMixed(a, b, mode=_lib.MIXED_3XTF32, ctx=ctx)
    assert st == 0 and rep["fell_back"] == 0, rep
    assert oracle.backward_error(a, x, b) <= max(n, 4) * 2.0 ** -53


@pytest.mark.parametrize("n", [544, 1100])
def test_ties_and_vanishing_columns(ctx, n):
    r = inputs.rng(61)
    a = np.where(r.random_sample((n, n)) < 0.5, -1.0, 1.0)  # every search of a chunk's first column is a tie
    a[512:, :40] = 0.0  # zero columns in every chunk but the first
    a += np.sqrt(n) * np.eye(n)
    b = r.standard_normal((n, 3))
    st, x, rep = L.MatrixLinEQSolveMixed(a, b, mode=_lib.MIXED_3XTF32, ctx=ctx)
    assert st == 0 and rep["fell_back"] == 0, rep
    assert oracle.backward_error(a, x, b) <= n * 2.0 ** -53
