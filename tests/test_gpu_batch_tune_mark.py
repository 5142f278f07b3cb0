"""The tuning table says of a mode-0 plan that nothing was timed, and of a mode-1 plan what was; both marks survive a
saved table."""
import pytest

from mrmath_b200 import _lib, inputs, linalg as L

pytestmark = pytest.mark.gpu


def test_untuned_plans_are_marked(tmp_path):
    _, _, mats, rhss = inputs.c5_batched(count=12, lo=8, hi=60, seed=4)
    c, d = _lib.Context(), _lib.Context()
    try:
        L.BatchLinEQSolve(mats, rhss, mode=0, ctx=c)
        assert L.batch_tune(c)["ms"] < 0
        L.BatchLinEQSolve(mats, rhss, mode=1, ctx=c)
        assert L.batch_tune(c)["ms"] > 0
        path = str(tmp_path / "tune.txt")
        L.batch_tune_save(path, ctx=c)
        assert sorted(float(line.split()[-1]) > 0 for line in open(path).read().splitlines()[1:]) == [False, True]
        assert L.batch_tune_load(path, ctx=d) == 2
        L.BatchLinEQSolve(mats, rhss, mode=0, ctx=d)
        assert L.batch_tune(d)["ms"] < 0
        L.BatchLinEQSolve(mats, rhss, mode=1, ctx=d)
        assert L.batch_tune(d)["ms"] > 0
    finally:
        c.close()
        d.close()
