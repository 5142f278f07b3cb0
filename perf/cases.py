"""The calls a program makes of this library, as cases that can be timed and compared.

A case is a dict of plain values with a "kind".  `prepare` makes its inputs from the seed alone, `run` is
one pass through the public entry points, `work` the bytes and operations the call cannot do without, and
`exact` the result in plain 64-bit torch / numpy.  `listed` holds the cases, `draw` gives more of the same
ranges.  Sizes and distributions are those of `mrmath_b200/inputs.py`, the tests and the benchmark, or
generic.
"""
import numpy as np
import torch

from mrmath_b200 import autograd, linalg as L

DEV = "cuda"

# one range per kind: the orders (or GEMM dimensions), then the right-hand sides
ORDERS = {
    "mult": (32, 4096), "ozaki": (256, 8192), "solve": (16, 6000), "factor": (32, 6000), "mixed": (500, 8192),
    "grad": (48, 4096), "batch": (200, 20000), "inverse": (16, 3000), "cholesky": (32, 6000), "complex": (8, 1000),
}
RHS = {"solve": (1, 16), "factor": (1, 16), "mixed": (1, 16), "grad": (1, 4), "cholesky": (1, 16), "complex": (1, 4)}


def listed():
    return [
        # one small product inside a larger computation: launch and latency
        {"name": "mult_small", "kind": "mult", "m": 128, "k": 128, "n": 128, "trans": 0, "op": L.DO_NONE},
        # an ordinary product of unpadded odd-sized matrices, second operand transposed, accumulated
        {"name": "mult_ragged", "kind": "mult", "m": 2999, "k": 1501, "n": 2777, "trans": 2, "op": L.DO_ADD},
        # the emulated FP64 product at the benchmark's size and element distribution
        {"name": "mult_ozaki", "kind": "ozaki", "m": 8192, "k": 8192, "n": 8192, "slices": 8},
        # the smallest systems: one solve of a few dozen unknowns, call after call
        {"name": "solve_small", "kind": "solve", "n": 100, "k": 1, "refine": 0},
        # the reference's own benchmark order (uniform [0, 1) system), with one refinement step
        {"name": "solve_1024", "kind": "solve", "n": 1024, "k": 1, "refine": 1},
        # factor once, substitute later: the drop-in pair of calls, odd order
        {"name": "factor_odd", "kind": "factor", "n": 2501, "k": 3},
        # the headline: mixed-precision solve of the benchmark system (the stopping rule bounds the backward
        # error, so the solution itself is fixed to about kappa times that: 4e-10 here, 2e-8 at kappa = 1e5)
        {"name": "mixed_8192", "kind": "mixed", "n": 8192, "k": 16, "kappa": 1e4},
        # a differentiable solve, forward and backward
        {"name": "grad_4096", "kind": "grad", "n": 4096, "k": 1},
        # many small uneven systems in one call
        {"name": "batch_20000", "kind": "batch", "count": 20000, "hi": 256, "mode": 0},
        # explicit inverse
        {"name": "inverse_1500", "kind": "inverse", "n": 1500},
        # symmetric positive definite system: Cholesky factor and solve
        {"name": "cholesky_3000", "kind": "cholesky", "n": 3000, "k": 4},
        # complex system; the complex entry points take host arrays
        {"name": "complex_600", "kind": "complex", "n": 600, "k": 2},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(sorted(ORDERS))
    lo, hi = ORDERS[kind]
    case = {"kind": kind}
    if kind in ("mult", "ozaki"):
        case.update({d: _log(rng, lo, hi) for d in ("m", "k", "n")})
        if kind == "mult":
            case.update(trans=rng.randrange(3), op=rng.choice((L.DO_NONE, L.DO_NONE, L.DO_ADD, L.DO_SUB)))
        else:
            case["slices"] = rng.choice((8, 8, 8, 6))
    elif kind == "batch":
        case.update(count=_log(rng, lo, hi), hi=rng.choice((32, 64, 100, 160, 256)), mode=rng.choice((0, 0, 1)))
    else:
        case["n"] = _log(rng, lo, hi)
        if kind in RHS:
            case["k"] = _log(rng, *RHS[kind])
        if kind == "solve":
            case["refine"] = rng.choice((0, 0, 1, 2))
        if kind == "mixed":
            case["kappa"] = rng.choice((1e2, 1e4))
    return case


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _batch_plan(case):
    """orders uniform in [8, hi], 1..4 right-hand sides, packed one after the other; a program that solves
    such a set again and again has the same orders each time"""
    r = np.random.RandomState(case["count"] + 1000 * case["hi"])
    n = r.randint(8, case["hi"] + 1, size=case["count"]).astype(np.int32)
    k = r.randint(1, 5, size=case["count"]).astype(np.int32)
    a_sz, b_sz = n.astype(np.int64) ** 2, n.astype(np.int64) * k
    a_off, b_off = np.cumsum(a_sz) - a_sz, np.cumsum(b_sz) - b_sz
    return n, k, a_off, b_off, int(a_sz.sum()), int(b_sz.sum())


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    s = {"case": case}
    if kind in ("mult", "ozaki"):
        m, k, n = case["m"], case["k"], case["n"]
        t = case.get("trans", 0)
        for name, shape in (("A", (k, m) if t == 1 else (m, k)), ("B", (n, k) if t == 2 else (k, n))):
            # g * 2^e, g Gaussian, e uniform in [-8, 8]
            e = torch.randint(-8, 9, shape, generator=g, device=DEV)
            s[name] = torch.ldexp(_randn(g, *shape), e)
        s["C"] = _randn(g, m, n)
    elif kind in ("solve", "factor", "inverse"):
        n, k = case["n"], case.get("k", 1)
        s["A"], s["B"] = _rand(g, n, n), _rand(g, n, k)
        s["X"] = torch.zeros_like(s["B"])
        s["LU"], s["indx"] = torch.empty_like(s["A"]), torch.zeros(n, dtype=torch.int32, device=DEV)
        s["status"] = torch.zeros(1, dtype=torch.int32, device=DEV)
    elif kind == "mixed":
        n = case["n"]
        u, _ = torch.linalg.qr(_randn(g, n, n))
        v, _ = torch.linalg.qr(_randn(g, n, n))
        sv = case["kappa"] ** (-torch.arange(n, dtype=torch.float64, device=DEV) / (n - 1))
        s["A"], s["B"] = ((u * sv) @ v.T).contiguous(), _randn(g, n, case["k"])
        s["X"] = torch.zeros_like(s["B"])
    elif kind == "grad":
        n = case["n"]
        s["A"] = (2.0 * _rand(g, n, n) - 1.0 + n * torch.eye(n, device=DEV, dtype=torch.float64)).requires_grad_()
        s["B"], s["W"] = _randn(g, n, case["k"]).requires_grad_(), _randn(g, n, case["k"])
    elif kind == "batch":
        n, k, a_off, b_off, na, nb = _batch_plan(case)
        A = 2.0 * _rand(g, na) - 1.0
        reps = torch.from_numpy(n.astype(np.int64)).to(DEV)
        first = torch.from_numpy(a_off).to(DEV).repeat_interleave(reps)
        order = reps.repeat_interleave(reps)
        i = torch.arange(order.numel(), device=DEV) - (torch.cumsum(reps, 0) - reps).repeat_interleave(reps)
        A[first + i * (order + 1)] += order.to(torch.float64)
        s.update(plan=(n, k, a_off, b_off), A=A, B=_randn(g, nb))
        s["X"] = torch.zeros_like(s["B"])
        s["info"] = torch.zeros(len(n), dtype=torch.int32, device=DEV)
    elif kind == "cholesky":
        n = case["n"]
        m = _rand(g, n, n) - 0.5
        s["A"] = m @ m.T + 0.25 * n * torch.eye(n, device=DEV, dtype=torch.float64)
        s["B"] = _rand(g, n, case["k"]) - 0.5
        s["X"], s["F"] = torch.zeros_like(s["B"]), torch.empty_like(s["A"])
        s["status"] = torch.zeros(1, dtype=torch.int32, device=DEV)
    elif kind == "complex":
        n, k = case["n"], case["k"]
        r = np.random.RandomState(seed % 2 ** 32)
        s["A"] = (r.random_sample((n, n)) - 0.5) + 1j * (r.random_sample((n, n)) - 0.5)
        s["B"] = (r.random_sample((n, k)) - 0.5) + 1j * (r.random_sample((n, k)) - 0.5)
    else:
        raise ValueError(kind)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "mult":
        # an accumulating product starts from a copy, so that every pass gives the same result
        dest = s["C"].clone() if case["op"] != L.DO_NONE else s["C"]
        L.dev_MatrixMultEx(dest, s["A"], s["B"], case["op"], case["trans"])
        return dest
    if kind == "ozaki":
        L.dev_MatrixMultOzaki(s["C"], s["A"], s["B"], case["slices"])
        return s["C"]
    if kind == "solve":
        L.dev_MatrixLinEQSolve(s["A"], s["B"], s["X"], case["refine"], s["status"])
        return s["X"], s["status"]
    if kind == "factor":
        s["LU"].copy_(s["A"])
        s["X"].copy_(s["B"])
        L.dev_MatrixLUDecompInPlace(s["LU"], s["indx"], s["status"])
        L.dev_MatrixLUBackSubst(s["LU"], s["indx"], s["X"])
        return s["LU"], s["indx"], s["X"], s["status"]
    if kind == "mixed":
        st, _ = L.dev_MatrixLinEQSolveMixed(s["A"], s["B"], s["X"])
        return s["X"], st
    if kind == "grad":
        x = autograd.solve(s["A"], s["B"])
        da, db = torch.autograd.grad(x, (s["A"], s["B"]), s["W"])
        return x, da, db
    if kind == "batch":
        L.dev_BatchLinEQSolve(*s["plan"], s["A"], s["B"], s["X"], s["info"], mode=case["mode"])
        return s["X"], s["info"]
    if kind == "inverse":
        s["LU"].copy_(s["A"])
        L.dev_MatrixInverseInPlace(s["LU"], s["status"])
        return s["LU"], s["status"]
    if kind == "cholesky":
        s["F"].copy_(s["A"])
        L.dev_MatrixCholeskyInPlace4(s["F"], s["status"])
        L.dev_MatrixCholeskySolveLinEq(s["F"], s["B"], s["X"])
        return s["F"], s["X"], s["status"]
    if kind == "complex":
        st, x = L.CplxMatrixLinEQSolve(s["A"], s["B"])
        return x, st
    raise ValueError(kind)


def work(case):
    kind = case["kind"]
    if kind in ("mult", "ozaki"):
        m, k, n = case["m"], case["k"], case["n"]
        c = 2 if case.get("op", L.DO_NONE) != L.DO_NONE else 1
        return {"bytes": 8 * (m * k + k * n + c * m * n), "flops": 2.0 * m * n * k}
    if kind == "batch":
        n, k, _, _, na, nb = _batch_plan(case)
        n, k = n.astype(np.float64), k.astype(np.float64)
        return {"bytes": 8 * (na + 2 * nb), "flops": float((2 / 3 * n ** 3 + 2 * n * n * k).sum())}
    n, k = case["n"], case.get("k", 1)
    if kind in ("solve", "mixed"):  # A and B in, X out
        r = case.get("refine", 0)
        return {"bytes": 8 * (n * n + 2 * n * k), "flops": 2 / 3 * n ** 3 + 2.0 * n * n * k * (1 + 2 * r)}
    if kind == "factor":  # the factors too
        return {"bytes": 8 * (2 * n * n + 2 * n * k), "flops": 2 / 3 * n ** 3 + 2.0 * n * n * k}
    if kind == "grad":  # dA too
        return {"bytes": 8 * (2 * n * n + 4 * n * k), "flops": 2 / 3 * n ** 3 + 6.0 * n * n * k}
    if kind == "inverse":
        return {"bytes": 16 * n * n, "flops": 2.0 * n ** 3}
    if kind == "cholesky":  # one triangle in and out
        return {"bytes": 8 * (n * n + 2 * n * k), "flops": 1 / 3 * n ** 3 + 2.0 * n * n * k}
    if kind == "complex":
        return {"bytes": 16 * (n * n + 2 * n * k), "flops": 8 / 3 * n ** 3 + 8.0 * n * n * k}
    raise ValueError(kind)


def _solve(a, b):
    """64-bit solve with one refinement step"""
    lu, p = torch.linalg.lu_factor(a)
    x = torch.linalg.lu_solve(lu, p, b)
    return x + torch.linalg.lu_solve(lu, p, b - a @ x)


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind in ("mult", "ozaki"):
        t, op = case.get("trans", 0), case.get("op", L.DO_NONE)
        p = (s["A"].T if t == 1 else s["A"]) @ (s["B"].T if t == 2 else s["B"])
        return p if op == L.DO_NONE else s["C"] + p if op == L.DO_ADD else s["C"] - p
    if kind == "solve":
        return _solve(s["A"], s["B"]), None
    if kind == "factor":
        lu, _ = torch.linalg.lu_factor(s["A"])
        return lu, None, _solve(s["A"], s["B"]), None
    if kind == "mixed":
        return _solve(s["A"], s["B"]), None
    if kind == "grad":
        a = s["A"].detach()
        x, db = _solve(a, s["B"].detach()), _solve(a.T, s["W"])
        return x, -db @ x.T, db
    if kind == "batch":
        n, k, a_off, b_off = s["plan"]
        x = torch.zeros_like(s["B"])
        for order in np.unique(n):  # one batched call per order and number of right-hand sides
            for rhs in np.unique(k[n == order]):
                at = np.nonzero((n == order) & (k == rhs))[0]
                ia = torch.from_numpy(a_off[at]).to(DEV)[:, None] + torch.arange(int(order) ** 2, device=DEV)
                ib = torch.from_numpy(b_off[at]).to(DEV)[:, None] + torch.arange(int(order) * int(rhs), device=DEV)
                y = torch.linalg.solve(s["A"][ia].view(len(at), order, order), s["B"][ib].view(len(at), order, rhs))
                x[ib] = y.reshape(len(at), -1)
        return x, None
    if kind == "inverse":
        return _solve(s["A"], torch.eye(case["n"], device=DEV, dtype=torch.float64)), None
    if kind == "cholesky":
        # the strict upper triangle is not written
        return torch.tril(torch.linalg.cholesky(s["A"])) + torch.triu(s["A"], 1), _solve(s["A"], s["B"]), None
    if kind == "complex":
        return np.linalg.solve(s["A"], s["B"]), None
    raise ValueError(kind)
