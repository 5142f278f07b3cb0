"""Batches that differ only in where their systems lie.  Each pair below has the same 64-bit plan signature (asserted),
so only a comparison of the plans themselves tells them apart: every call must read and write at its own offsets."""
import numpy as np
import pytest

import oracle
from mrmath_b200 import linalg as L

FAR = 2 ** 24
# (orders, right-hand sides, offsets of A, offsets of B) twice
PAIRS = [
    (([8], [1], [0], [0]), ([8], [1], [0], [FAR])),
    (([8], [1], [2 ** 20], [0]), ([8], [1], [0], [1])),
    (([9, 40], [2, 1], [0, 81], [0, 18]), ([9, 40], [2, 1], [0, 81], [FAR, FAR + 18])),
]


def signature(plan, mode):
    sig = 1469598103934665603 ^ mode
    for n, k, a, b in zip(*plan):
        sig = (sig ^ (n * 16 + k) ^ (a << 20) ^ (b << 40)) % 2 ** 64 * 1099511628211 % 2 ** 64
    return sig


@pytest.mark.gpu
@pytest.mark.parametrize("pair", range(len(PAIRS)))
@pytest.mark.parametrize("mode", [0, 1])
def test_plans_that_share_a_signature(ctx, pair, mode):
    import torch
    first, second = PAIRS[pair]
    assert signature(first, mode) == signature(second, mode)
    r = np.random.RandomState(pair)
    A = torch.zeros(2 ** 20 + 2048, dtype=torch.float64, device="cuda")
    B = torch.zeros(FAR + 2048, dtype=torch.float64, device="cuda")
    X = torch.empty_like(B)
    for plan in (first, second, first, second):
        n, k, a_off, b_off = (np.array(v, dtype) for v, dtype in zip(plan, (np.int32, np.int32, np.int64, np.int64)))
        mats = [2.0 * r.random_sample((q, q)) - 1.0 + q * np.eye(q) for q in n]
        rhss = [r.standard_normal((q, c)) for q, c in zip(n, k)]
        A.zero_()
        B.zero_()
        X.fill_(7.0)
        for a, b, ao, bo in zip(mats, rhss, a_off, b_off):
            A[ao:ao + a.size] = torch.from_numpy(a.ravel()).cuda()
            B[bo:bo + b.size] = torch.from_numpy(b.ravel()).cuda()
        info = torch.full((len(n),), 9, dtype=torch.int32, device="cuda")
        L.dev_BatchLinEQSolve(n, k, a_off, b_off, A, B, X, info, mode=mode, ctx=ctx)
        assert not info.any()
        for a, b, bo in zip(mats, rhss, b_off):
            x = X[bo:bo + b.size].cpu().numpy().reshape(b.shape)
            assert oracle.backward_error(a, x, b) <= 4 * a.shape[0] * 2.0 ** -53
            X[bo:bo + b.size] = 7.0
        assert bool((X == 7.0).all())  # nothing else was written
