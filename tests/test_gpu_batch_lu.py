"""FP64 batched solves at the edges of their code: leaves of 32 and 16 columns, one, two or four systems a
thread block, every count of right-hand sides, ties, scales outside the reciprocal's range, singular systems."""
import numpy as np
import pytest
import scipy.linalg

import oracle
from mrmath_b200 import inputs, linalg as L

pytestmark = pytest.mark.gpu

EDGE = [1, 2, 8, 9, 15, 16, 17, 31, 32, 33, 47, 48, 63, 64, 65, 96, 127, 128, 129, 159, 161, 225, 255, 256]


def _check(a, b, x):
    # Gaussian elimination's backward error is a small multiple of n u times the growth of the factors
    n = a.shape[0]
    growth = np.abs(np.triu(scipy.linalg.lu_factor(a, check_finite=False)[0])).max() / np.abs(a).max()
    eta = oracle.backward_error(a, x, b)
    assert eta <= 4 * n * 2.0 ** -53 * max(1.0, growth), (n, b.shape[1], eta)


def _hadamard(n):
    h = np.ones((1, 1))
    while h.shape[0] < n:
        h = np.block([[h, h], [h, -h]])
    return h


@pytest.mark.parametrize("repeat", [1, 3])  # few systems (all warps on each); more than the GPU holds at once
def test_edge_orders(ctx, repeat):
    r = inputs.rng(41 + repeat)
    mats, rhss = [], []
    for _ in range(repeat):
        for n in EDGE:
            for k in range(1, 9):
                mats.append(2.0 * r.random_sample((n, n)) - 1.0)
                rhss.append(r.standard_normal((n, k)))
    xs, info, _ = L.BatchLinEQSolve(mats, rhss, mode=0, ctx=ctx)
    assert np.all(info == 0)
    for a, b, x in zip(mats, rhss, xs):
        _check(a, b, x)


@pytest.mark.parametrize("repeat", [1, 40])
def test_ties_scales_and_singular(ctx, repeat):
    r = inputs.rng(43)
    mats, rhss, scale, singular = [], [], [], []

    def add(a, b, s=0, sing=0):
        mats.append(np.ascontiguousarray(a))
        rhss.append(np.ascontiguousarray(b))
        scale.append(s)
        singular.append(sing)

    for n in (16, 32, 64, 128, 256):  # every pivot search is a tie
        h = _hadamard(n)
        add(h[r.permutation(n)][:, r.permutation(n)], r.standard_normal((n, 3)))
    for n in (5, 40, 130, 256):  # diagonals of U beyond 2^1000 and below 2^-1000
        for e in (1005, -1005):
            a = 2.0 * r.random_sample((n, n)) - 1.0 + n * np.eye(n)
            add(np.ldexp(a, e), np.ldexp(r.standard_normal((n, 2)), e), e)
    for n in (3, 33, 100, 200):  # a column that vanishes, a NaN column
        a = r.random_sample((n, n))
        a[:, n // 2] = 0.0
        add(a, np.ones((n, 1)), sing=1)
        a = r.random_sample((n, n))
        a[:, n - 1] = np.nan
        add(a, np.ones((n, 8)), sing=1)
    mats, rhss, scale, singular = mats * repeat, rhss * repeat, scale * repeat, singular * repeat
    xs, info, _ = L.BatchLinEQSolve(mats, rhss, mode=0, ctx=ctx)
    assert list(info) == singular
    for a, b, x, e, sing in zip(mats, rhss, xs, scale, singular):
        if not sing:
            _check(np.ldexp(a, -e), np.ldexp(b, -e), x)
