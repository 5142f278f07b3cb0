"""The emulated product's slices: the result against the scheme carried out on the CPU with whole numbers, for every
kind of entry the slicing treats apart (zeros, signs, powers of two, tiny and huge rows, more than eight slices)."""
import numpy as np
import pytest
import torch

from mrmath_b200 import inputs, linalg as L

pytestmark = pytest.mark.gpu


def _slices(x, axis, s):
    """exponents along `axis` and the s whole-number slices, by the defining steps"""
    m = np.abs(x).max(axis=axis, keepdims=True)
    e = np.where(m > 0, np.frexp(m)[1], 0)
    v = x * np.ldexp(1.0, -e)
    out = []
    for _ in range(s):
        v = v * 128.0
        d = np.trunc(v)
        v = v - d
        out.append(d.astype(np.int64))
    return e, out


def _scheme(a, b, s):
    """the product and the sum of the magnitudes of its terms"""
    ea, pa = _slices(a, 1, s)
    eb, pb = _slices(b, 0, s)
    c, mag = np.zeros((a.shape[0], b.shape[1])), np.zeros((a.shape[0], b.shape[1]))
    for d in range(2, s + 2):
        t = sum(pa[p - 1] @ pb[d - p - 1] for p in range(1, d) if p <= s and d - p <= s)
        c += np.ldexp(t.astype(np.float64), -7 * d)  # (exact: whole numbers below 2^53)
        mag += np.abs(np.ldexp(t.astype(np.float64), -7 * d))
    return np.ldexp(c, ea + eb), np.ldexp(mag, ea + eb)


def _matrix(r, m, k):
    x = r.standard_normal((m, k)) * np.exp2(r.randint(-40, 1, size=(m, k)))
    x[r.random_sample((m, k)) < 0.1] = 0.0
    x = np.where(r.random_sample((m, k)) < 0.1, np.sign(x) * np.exp2(r.randint(-20, 1, size=(m, k))), x)
    scale = np.exp2(r.choice([-900, -3, 0, 5, 300], size=(m, 1)))
    x = x * scale
    if m > 2:
        x[m // 2] = 0.0
    return x


@pytest.mark.parametrize("s", [2, 5, 8, 9, 10])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (5, 3, 9), (33, 130, 31), (64, 127, 65), (70, 257, 100), (3, 600, 40)])
def test_scheme(ctx, m, k, n, s):
    r = inputs.rng(m + k + n + s)
    a, b = _matrix(r, m, k), np.ascontiguousarray(_matrix(r, n, k).T)
    want, mag = _scheme(a, b, s)
    # odd strides and an odd first element: rows that start off the 16-byte boundary
    A = torch.zeros(m * (k + 1) + 1, dtype=torch.float64, device="cuda")[1:].as_strided((m, k), (k + 1, 1))
    B = torch.zeros(k * (n + 2) + 1, dtype=torch.float64, device="cuda")[1:].as_strided((k, n), (n + 2, 1))
    A.copy_(torch.from_numpy(a)), B.copy_(torch.from_numpy(b))
    for got in (L.MatrixMultOzaki(a, b, slices=s, ctx=ctx), _device(ctx, A, B, s)):
        # s sums in FP64 of exact terms, and the scaling's two roundings
        assert np.all(np.abs(got - want) <= (s + 3) * 2.0 ** -53 * mag)


def _device(ctx, A, B, s):
    C = torch.zeros((A.shape[0], B.shape[1]), dtype=torch.float64, device="cuda")
    L.dev_MatrixMultOzaki(C, A, B, slices=s, ctx=ctx)
    return C.cpu().numpy()
