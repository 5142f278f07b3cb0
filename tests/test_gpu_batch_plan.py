"""The batched solve's plan stays on the device between calls: routines that run in between must not
touch it.  (The Ozaki product and the product's error report once shared its workspace, and the next
call with the same plan read their data as orders and offsets.)"""
import numpy as np
import pytest

from mrmath_b200 import inputs, linalg as L

pytestmark = pytest.mark.gpu


def test_plan_survives_other_calls(ctx):
    _, _, mats, rhss = inputs.c5_batched(count=40, lo=8, hi=100, seed=3)
    first, info, _ = L.BatchLinEQSolve(mats, rhss, ctx=ctx)
    assert not info.any()
    r = np.random.RandomState(1)
    a, b = r.standard_normal((300, 200)), r.standard_normal((200, 150))
    for between in (lambda: L.MatrixMultOzaki(a, b, ctx=ctx),
                    lambda: L.MatrixMultErrorReport(L.MatrixMult(a, b, ctx=ctx), a, b, ctx=ctx),
                    lambda: L.MatrixLinEQSolveMixed(r.random_sample((300, 300)) + 3 * np.eye(300), r.random_sample((300, 2)), ctx=ctx),
                    lambda: L.MatrixInverseInPlace(r.random_sample((90, 90)), ctx=ctx)):
        between()
        again, info, _ = L.BatchLinEQSolve(mats, rhss, ctx=ctx)
        assert not info.any()
        for x, y in zip(first, again):
            assert np.array_equal(x, y)
