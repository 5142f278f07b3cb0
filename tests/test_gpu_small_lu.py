"""Orders up to 256 in one launch, and 257 .. 512 in linked leaves, against the general recursion (which a call with
progress reports takes) and the oracle: factors, interchanges, solves, inverse, over strides, offsets, ties, scales."""
import numpy as np
import pytest
import torch

import oracle
from mrmath_b200 import _lib, inputs, linalg as L

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
EDGE = [1, 2, 3, 8, 9, 31, 32, 33, 63, 64, 65, 97, 127, 128, 129, 160, 224, 225, 255, 256, 257, 288, 300, 511, 512]


@pytest.fixture(scope="module")
def plain():
    """a context whose calls take the recursion"""
    c = _lib.Context()
    c.set_progress(lambda pct: None)
    yield c
    c.set_progress(None)


def _strided(a, pad, shift):
    """a on the device, `pad` unused elements after each row, `shift` elements past an aligned address"""
    n, k = a.shape
    buf = torch.full((n * (k + pad) + shift,), 7.0, dtype=torch.float64, device="cuda")
    view = buf[shift:].as_strided((n, k), (k + pad, 1))
    view.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return buf, view


def _factor(ctx, a, pad, shift):
    buf, f = _strided(a, pad, shift)
    idx = torch.zeros(a.shape[0], dtype=torch.int32, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    L.dev_MatrixLUDecompInPlace(f, idx, st, ctx=ctx)
    torch.cuda.synchronize()
    n = a.shape[0]
    if pad:
        rest = buf[shift:][: n * (n + pad)].view(n, n + pad)[:, n:]
        assert torch.all(rest == 7.0)  # the unused elements stay
    return int(st.item()), f.cpu().numpy(), idx.cpu().numpy()


def _error(a, lu, idx):
    pa = a.copy()
    for i, q in enumerate(idx):
        if q != i:
            pa[[i, q]] = pa[[q, i]]
    lo, up = np.tril(lu, -1) + np.eye(a.shape[0]), np.triu(lu)
    return np.abs(lo @ up - pa).max() / (np.abs(lo) @ np.abs(up)).max()


@pytest.mark.parametrize("n", EDGE)
@pytest.mark.parametrize("pad,shift", [(0, 0), (1, 0), (2, 0), (3, 1)])
def test_factor_forms(ctx, plain, n, pad, shift):
    a = 2.0 * inputs.rng(n).random_sample((n, n)) - 1.0
    st, lu, idx = _factor(ctx, a, pad, shift)
    st0, lu0, idx0 = _factor(plain, a, pad, shift)
    assert st == st0 == 0 and np.array_equal(idx, idx0)
    # |L U - P A| <= n u |L| |U| (the products of the unit-lower triangle add one rounding)
    assert max(_error(a, lu, idx), _error(a, lu0, idx0)) <= (n + 1) * U


@pytest.mark.parametrize("n,k", [(1, 1), (5, 8), (31, 9), (64, 16), (100, 1), (129, 7), (200, 17), (256, 64), (256, 70), (400, 3)])
@pytest.mark.parametrize("refine", [0, 1])
def test_solve(ctx, plain, n, k, refine):
    r = inputs.rng(n + k)
    a, b = 2.0 * r.random_sample((n, n)) - 1.0, r.standard_normal((n, k))
    growth = max(1.0, np.abs(np.triu(_factor(ctx, a, 0, 0)[1])).max() / np.abs(a).max())
    A, (_, B) = torch.from_numpy(a).cuda(), _strided(b, 1, 1)
    for c in (ctx, plain):
        X = torch.empty((n, k), dtype=torch.float64, device="cuda")
        L.dev_MatrixLinEQSolve(A, B, X, refine, ctx=c)
        assert oracle.backward_error(a, X.cpu().numpy(), b) <= 4 * n * U * growth


@pytest.mark.parametrize("n", [32, 64, 128, 256, 512])
def test_ties(ctx, n):
    h = np.ones((1, 1))
    while h.shape[0] < n:
        h = np.block([[h, h], [h, -h]])
    # rows of a Hadamard matrix in any order: multipliers 0 or +-1, exact, every search a tie
    a = h[inputs.rng(n).permutation(n)]
    ref = a.copy()
    rc, i0 = oracle.lu_decomp_inplace(ref)
    st, lu, idx = _factor(ctx, a, 0, 0)
    assert st == rc == 0 and np.array_equal(idx, i0) and np.array_equal(lu, ref)


@pytest.mark.parametrize("n", [3, 40, 129, 256])
def test_singular_and_scales(ctx, n):
    r = inputs.rng(n)
    for bad in (0.0, np.nan):
        a = r.random_sample((n, n))
        a[:, n // 2] = bad
        assert _factor(ctx, a, 0, 0)[0] == 1
        inv = torch.from_numpy(a).cuda()
        st = torch.zeros(1, dtype=torch.int32, device="cuda")
        L.dev_MatrixInverseInPlace(inv, st, ctx=ctx)
        assert int(st.item()) == 1
        assert L.MatrixLinEQSolve(a, np.ones((n, 1)), ctx=ctx)[0] == 1
    a, b = 2.0 * r.random_sample((n, n)) - 1.0 + n * np.eye(n), r.standard_normal((n, 2))
    for e in (1005, -1005):  # diagonals outside the reciprocal's range
        A, B = torch.from_numpy(np.ldexp(a, e)).cuda(), torch.from_numpy(np.ldexp(b, e)).cuda()
        X = torch.empty_like(B)
        L.dev_MatrixLinEQSolve(A, B, X, ctx=ctx)
        assert oracle.backward_error(a, X.cpu().numpy(), b) <= 4 * n * U


def test_capture_after_a_larger_call():
    c = _lib.Context()
    n, k = 100, 2
    r = inputs.rng(5)
    big = torch.from_numpy(r.random_sample((600, 600))).cuda()
    L.dev_MatrixLinEQSolve(big, big[:, :8].contiguous(), torch.empty((600, 8), dtype=torch.float64, device="cuda"), ctx=c)
    a, b = r.random_sample((n, n)) + np.eye(n), r.standard_normal((n, k))
    A, B = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    X = torch.zeros_like(B)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        L.dev_MatrixLinEQSolve(A, B, X, ctx=c)
    for _ in range(2):
        X.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert oracle.backward_error(a, X.cpu().numpy(), b) <= 64 * n * U
    del g
