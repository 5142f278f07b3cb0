"""The product's tile shapes (128, 64, 32 and 32 x 16) at their edges, every operand layout and
destination operation, destinations with even and odd row strides, and the repacking copy.

Bound: each element is a sum of K products accumulated in FP64, so it is within (K + 2) 2^-53 times
the sum of their magnitudes (plus the old value's) of the product in exact arithmetic, which long
double gives to 2^-64; one more 2^-53 covers the reference's rounding to double."""
import numpy as np
import pytest

from mrmath_b200 import linalg as L

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (31, 15, 16), (32, 16, 17), (33, 17, 40), (64, 64, 15), (65, 1, 300), (129, 127, 33),
          (200, 16, 64), (257, 300, 48), (700, 650, 100), (1500, 1300, 20), (2100, 2050, 17)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("trans", [0, 1, 2])
def test_tile_shapes(ctx, m, n, k, trans):
    import torch
    r = np.random.RandomState(m * 7 + n * 3 + k + trans)
    a, b, c0 = r.standard_normal((m, k)), r.standard_normal((k, n)), r.standard_normal((m, n))

    def on_device(x):  # (a one-row array may carry any row stride: the tensor is made with its own)
        t = torch.empty(x.shape, dtype=torch.float64, device="cuda")
        t.copy_(torch.from_numpy(x.copy()))
        return t

    A, B = on_device(a.T if trans == 1 else a), on_device(b.T if trans == 2 else b)
    rows = np.unique(np.concatenate([np.arange(min(m, 40)), r.randint(0, m, 40), np.arange(max(0, m - 40), m)]))
    prod = (a[rows].astype(np.longdouble)) @ b.astype(np.longdouble)
    mag = np.abs(a[rows]) @ np.abs(b)
    for op in (L.DO_NONE, L.DO_ADD, L.DO_SUB):
        for pad in (0, 1, 2):  # destination row strides n, n + 1, n + 2
            buf = torch.full((m, n + pad), 7.0, dtype=torch.float64, device="cuda")
            C = buf[:, :n]
            C.copy_(torch.from_numpy(c0))
            L.dev_MatrixMultEx(C, A, B, op, trans, ctx=ctx)
            torch.cuda.synchronize()
            got = buf.cpu().numpy()
            assert np.all(got[:, n:] == 7.0)
            old = 0.0 if op == L.DO_NONE else c0[rows]
            want = old + prod if op != L.DO_SUB else old - prod
            bound = (k + 3) * 2.0 ** -53 * (mag + np.abs(old))
            assert np.all(np.abs(got[rows, :n] - want) <= bound), (op, pad)


@pytest.mark.parametrize("rows,cols", [(1, 1), (31, 63), (32, 64), (33, 65), (3, 257), (300, 129)])
@pytest.mark.parametrize("pad", [0, 1, 2])
def test_repacked_operand(ctx, rows, cols, pad):
    """A product with the identity gives the operand back exactly, through the copy where the rows or
    the base are not 16-byte aligned."""
    import torch
    buf = torch.randn((rows + 1, cols + pad), dtype=torch.float64, device="cuda")
    for view in (buf[:rows, :cols], buf[1:, :cols]):
        eye = torch.eye(cols, dtype=torch.float64, device="cuda")
        out = torch.empty((rows, cols), dtype=torch.float64, device="cuda")
        L.dev_MatrixMultEx(out, view, eye, ctx=ctx)
        torch.cuda.synchronize()
        assert torch.equal(out, view)
