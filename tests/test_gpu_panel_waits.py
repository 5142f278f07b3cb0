"""Waits inside a panel's cluster that run out (a poll limit of 0, and of a few): the call ends with B2M_ERR_TIMEOUT or
with the right result, never with rows that are not the matrix's, and the context then works as before."""
import numpy as np
import pytest

from mrmath_b200 import _lib, inputs, linalg as L

pytestmark = pytest.mark.gpu


def _ends(c, call, same):
    """`call` under short limits, then with the built-in one"""
    want = call()
    for polls in (0, 1, 2, 5, 30, 0):
        c.set_wait_limit(polls)
        try:
            got = call()
            assert polls > 0 and same(got, want)
        except _lib.B2MError as e:
            assert e.status == _lib.ERR_TIMEOUT
        c.set_wait_limit(-1)
        assert same(call(), want)


@pytest.mark.parametrize("n", [513, 1024, 1500])  # (up to 512 rows a panel is one CTA, without waits)
@pytest.mark.parametrize("graphs", [True, False])
def test_linked_leaves(n, graphs):
    c = _lib.Context()
    try:
        c.use_graphs(graphs)
        a = 2.0 * inputs.rng(n).random_sample((n, n)) - 1.0

        def call():
            st, lu, idx = L.MatrixLUDecomp(a, ctx=c)
            assert st == 0
            return lu, idx

        _ends(c, call, lambda x, y: np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1]))
    finally:
        c.close()


@pytest.mark.parametrize("n", [8200, 16400])  # leaves of 16 and 8 columns
def test_tall_panels(n):
    import torch
    c = _lib.Context()
    try:
        g = torch.Generator(device="cuda").manual_seed(n)
        a = 2.0 * torch.rand((n, n), generator=g, device="cuda", dtype=torch.float64) - 1.0

        def call():
            lu, idx = a.clone(), torch.zeros(n, dtype=torch.int32, device="cuda")
            st = torch.zeros(1, dtype=torch.int32, device="cuda")
            L.dev_MatrixLUDecompInPlace(lu, idx, st, ctx=c)
            torch.cuda.synchronize()
            if int(st.item()) != 0:
                raise _lib.B2MError(int(st.item()), "")
            return lu, idx

        _ends(c, call, lambda x, y: torch.equal(x[0], y[0]) and torch.equal(x[1], y[1]))
    finally:
        c.close()


@pytest.mark.parametrize("n", [300, 600, 1300])
def test_complex_panels(n):
    c = _lib.Context()
    try:
        r = inputs.rng(n)
        a = (r.random_sample((n, n)) - 0.5) + 1j * (r.random_sample((n, n)) - 0.5)

        def call():
            lu = a.copy()
            st, idx = L.CplxMatrixLUDecompInPlace(lu, ctx=c)
            assert st == 0
            return lu, idx

        _ends(c, call, lambda x, y: np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1]))
    finally:
        c.close()
