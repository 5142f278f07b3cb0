"""The product's 128 x 128 tile, at its edges: every operand layout and destination operation, destinations with even and
odd row strides, through the prefetch of the old values and both epilogues.

12 x 12 tiles of 128 are one wave of 148 SMs and 23 or 24 tiles of 64 each way are two waves of pairs, so by the
estimates of pick_tile (9 + 0.139 K against 5 + 0.152 K) these shapes take the large tile from K = 309 on.  Bound: a sum
of K products in FP64 is within (K + 2) 2^-53 times the sum of their magnitudes (plus the old value's) of the exact one,
which long double gives to 2^-64; one more 2^-53 covers its rounding to double."""
import numpy as np
import pytest

from mrmath_b200 import linalg as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1536, 1536, 320), (1409, 1535, 333), (1473, 1410, 400), (1535, 1409, 401)])
@pytest.mark.parametrize("trans", [0, 1, 2])
def test_edges(ctx, m, n, k, trans):
    import torch
    r = np.random.RandomState(m + n + k + trans)
    a, b, c0 = r.standard_normal((m, k)), r.standard_normal((k, n)), r.standard_normal((m, n))
    A = torch.from_numpy(np.ascontiguousarray(a.T if trans == 1 else a)).cuda()
    B = torch.from_numpy(np.ascontiguousarray(b.T if trans == 2 else b)).cuda()
    # rows across a tile's warps and at the matrix's end; every column
    rows = np.unique(np.concatenate([np.arange(0, 130, 9), r.randint(0, m, 10), np.arange(m - 6, m)]))
    prod = a[rows].astype(np.longdouble) @ b.astype(np.longdouble)
    mag = np.abs(a[rows]) @ np.abs(b)
    for op in (L.DO_NONE, L.DO_ADD, L.DO_SUB):
        for pad in (0, 1, 2):
            buf = torch.full((m, n + pad), 7.0, dtype=torch.float64, device="cuda")
            C = buf[:, :n]
            C.copy_(torch.from_numpy(c0))
            L.dev_MatrixMultEx(C, A, B, op, trans, ctx=ctx)
            torch.cuda.synchronize()
            got = buf.cpu().numpy()
            assert np.all(got[:, n:] == 7.0)
            old = 0.0 if op == L.DO_NONE else c0[rows]
            want = old + prod if op != L.DO_SUB else old - prod
            assert np.all(np.abs(got[rows, :n] - want) <= (k + 3) * 2.0 ** -53 * (mag + np.abs(old))), (op, pad)
