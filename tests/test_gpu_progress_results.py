"""A progress callback changes nothing but the reports: factors, interchanges and solutions have the same bits with and
without one, at every order where the factorisation's form changes.  The recursion, which the allocation-free solve
takes, is held against the oracle at the same orders."""
import numpy as np
import pytest
import torch

import oracle
from mrmath_b200 import _lib, inputs, linalg as L

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 8, 31, 32, 33, 64, 65, 100, 127, 128, 129, 225, 255, 256, 257, 300, 511, 512, 513, 700]


@pytest.mark.parametrize("n", ORDERS)
def test_same_bits_with_reports(ctx, n):
    a, b = inputs.rng(n).random_sample((n, n)), inputs.rng(n).standard_normal((n, 3))
    c = _lib.Context()
    seen = []
    try:
        c.set_progress(seen.append)
        st, lu, idx = L.MatrixLUDecomp(a, ctx=c)
        assert seen == [min(n, j + 32) * 100 // n for j in range(0, n, 32)]
        x = L.MatrixLinEQSolve(a, b, ctx=c)[1]
        c.set_progress(None)
    finally:
        c.close()
    st0, lu0, idx0 = L.MatrixLUDecomp(a, ctx=ctx)
    assert st == st0 == 0 and np.array_equal(idx, idx0) and np.array_equal(lu, lu0)
    assert np.array_equal(x, L.MatrixLinEQSolve(a, b, ctx=ctx)[1])
    ref = a.copy()
    rc, i0 = oracle.lu_decomp_inplace(ref)
    assert rc == 0 and np.array_equal(idx, i0)


@pytest.mark.parametrize("n", [n for n in ORDERS if n <= 512])
def test_recursion(n):
    a, b = inputs.rng(n).random_sample((n, n)), inputs.rng(n).standard_normal((n, 3))
    A, B = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    X, st = torch.empty_like(B), torch.full((1,), 7, dtype=torch.int32, device="cuda")
    assert _lib.lib.b2m_dev_MatrixLinEQSolveNoAlloc(
        torch.cuda.current_stream().cuda_stream, A.data_ptr(), A.stride(0) * 8, n, B.data_ptr(), B.stride(0) * 8,
        X.data_ptr(), X.stride(0) * 8, 3, st.data_ptr()) == _lib.OK
    ref = a.copy()
    oracle.lu_decomp_inplace(ref)
    growth = max(1.0, np.abs(np.triu(ref)).max() / np.abs(a).max())
    assert int(st.item()) == 0 and oracle.backward_error(a, X.cpu().numpy(), b) <= 4 * n * 2.0 ** -53 * growth
