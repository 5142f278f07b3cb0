"""The allocation-free solve allocates nothing: free device memory stays as it was over many calls, and a call can be
captured into a graph (where an allocation or a new stream of its own would fail)."""
import numpy as np
import pytest
import torch

import oracle
from mrmath_b200 import _lib, inputs

pytestmark = pytest.mark.gpu


def _solve(A, B, X, st):
    rc = _lib.lib.b2m_dev_MatrixLinEQSolveNoAlloc(
        torch.cuda.current_stream().cuda_stream, A.data_ptr(), A.stride(0) * 8, A.shape[0], B.data_ptr(),
        B.stride(0) * 8, X.data_ptr(), X.stride(0) * 8, B.shape[1], st.data_ptr())
    assert rc == _lib.OK


@pytest.mark.parametrize("n,k", [(64, 3), (200, 64), (257, 1), (300, 5), (384, 64), (512, 64)])
def test_no_growth_and_capture(n, k):
    r = inputs.rng(n)
    a, b = 2.0 * r.random_sample((n, n)) - 1.0 + np.sqrt(n) * np.eye(n), r.standard_normal((n, k))
    A, B = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    X, st = torch.zeros_like(B), torch.zeros(1, dtype=torch.int32, device="cuda")
    _solve(A, B, X, st)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(64):
        _solve(A, B, X, st)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _solve(A, B, X, st)
    X.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert int(st.item()) == 0 and oracle.backward_error(a, X.cpu().numpy(), b) <= 4 * n * 2.0 ** -53
    del g
