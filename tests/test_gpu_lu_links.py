"""The pieces between the FP64 LU's leaves: the permutation built from an interchange vector, and
factorisations whose orders put the outer panels' triangular solve and the linked leaves at their
edges."""
import numpy as np
import pytest

import oracle
from mrmath_b200 import linalg as L

pytestmark = pytest.mark.gpu


def interchange(n, kind, seed):
    r = np.random.RandomState(seed)
    i = np.arange(n)
    if kind == "lapack":
        return (i + r.randint(0, n, n) % (n - i)).astype(np.int32)
    if kind == "last":
        return np.full(n, n - 1, np.int32)
    if kind == "next":
        return np.minimum(i + 1, n - 1).astype(np.int32)
    if kind == "none":
        return i.astype(np.int32)
    return r.randint(-2, n + 2, n).astype(np.int32)  # reaching back, and out of range (ignored)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 500, 1023, 1025, 4097])
@pytest.mark.parametrize("kind", ["lapack", "last", "next", "none", "any"])
def test_permutation_of_an_interchange_vector(ctx, n, kind):
    """With the identity as factors the back substitution returns the permuted right-hand side."""
    import torch
    ipiv = interchange(n, kind, n)
    want = np.arange(n)
    for i, q in enumerate(ipiv):
        if 0 <= q < n:
            want[i], want[q] = want[q], want[i]
    lu = torch.eye(n, dtype=torch.float64, device="cuda")
    x = torch.arange(n, dtype=torch.float64, device="cuda").reshape(n, 1).repeat(1, 2).contiguous()
    L.dev_MatrixLUBackSubst(lu, torch.from_numpy(ipiv).cuda(), x, ctx=ctx)
    torch.cuda.synchronize()
    assert np.array_equal(x.cpu().numpy()[:, 0], want)
    assert np.array_equal(x.cpu().numpy()[:, 1], want)


@pytest.mark.parametrize("n", [513, 519, 545, 575, 640, 767, 769, 800, 1793])
def test_factors_at_the_edges(ctx, n):
    """Orders around the leaf (32) and outer panel (256) widths, rows and columns of mixed scale, so that
    interchanges reach everywhere."""
    r = np.random.RandomState(n)
    a = r.standard_normal((n, n)) * 2.0 ** r.randint(-3, 4, (n, 1))
    ref, got = a.copy(), a.copy()
    rc, idx = oracle.lu_decomp_inplace(ref)
    st, piv = L.MatrixLUDecompInPlace(got, ctx=ctx)
    assert rc == st == 0
    assert np.array_equal(piv, idx)
    assert np.linalg.norm(got - ref) <= 1e-12 * np.linalg.norm(ref)
    b = r.standard_normal((n, 3))
    x = b.copy()
    L.MatrixLUBackSubst(got, piv, x, ctx=ctx)
    assert oracle.backward_error(a, x, b) <= n * 2.0 ** -53
