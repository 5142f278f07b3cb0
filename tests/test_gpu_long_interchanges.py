"""Interchange vectors of more than 32768 entries, around the orders where the permutation's kernel changes (three tables
of 16 bits in shared memory, one of 32 bits, global memory)."""
import numpy as np
import pytest

from mrmath_b200 import linalg as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32768, 32769, 58112, 58113])
@pytest.mark.parametrize("kind", ["lapack", "any"])
def test_permutation(ctx, n, kind):
    """With the identity as factors the back substitution returns the permuted right-hand side."""
    import torch
    r = np.random.RandomState(n)
    i = np.arange(n)
    ipiv = (i + r.randint(0, n, n) % (n - i) if kind == "lapack" else r.randint(-2, n + 2, n)).astype(np.int32)
    want = np.arange(n)
    for j, q in enumerate(ipiv):
        if 0 <= q < n:
            want[j], want[q] = want[q], want[j]
    lu = torch.eye(n, dtype=torch.float64, device="cuda")
    x = torch.arange(n, dtype=torch.float64, device="cuda").reshape(n, 1).repeat(1, 2).contiguous()
    L.dev_MatrixLUBackSubst(lu, torch.from_numpy(ipiv).cuda(), x, ctx=ctx)
    torch.cuda.synchronize()
    assert np.array_equal(x.cpu().numpy()[:, 0], want)
    assert np.array_equal(x.cpu().numpy()[:, 1], want)
