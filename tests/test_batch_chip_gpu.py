"""The batched solve with vectors in shared memory (csrc/batch.cu) at the sizes
where a system's arrays move: one row, rows short of a thread each, the matrix
on chip and not, the correction and the product in global memory, vectors
that do not fit, 4-byte columns."""
import numpy as np
import pytest

from seldon_b200 import matgen
from tests.helpers import to_dev, to_host

pytestmark = pytest.mark.gpu

# sides of the systems of one batch (rows = side^2)
BATCHES = [[1, 2, 3, 5, 11, 22], [8, 31, 45, 46], [3, 67, 68, 95, 106], [119, 120, 121, 17],
           [138, 139, 140, 141, 1], [257, 30, 4]]


@pytest.mark.parametrize("sides", BATCHES, ids=[str(max(b)) for b in BATCHES])
@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("guess", [False, True])
def test_chip_solves(cuda, sides, mixed, guess):
    import torch
    from seldon_b200 import api
    rng = np.random.default_rng(sum(sides))
    systems = [matgen.lap2d(g, shift=0.01) for g in sides]
    xs = [rng.uniform(-1, 1, g * g) for g in sides]
    rhs = [matgen.matvec(*s, x) for s, x in zip(systems, xs)]
    rhs[-1][:] = 0.0  # a zero right-hand side leaves its x untouched
    B = api.Batch(systems)
    x0 = np.concatenate([rng.uniform(-1, 1, x.size) for x in xs])
    sols = []
    for _ in range(2):
        X = to_dev(x0)
        it = torch.zeros(B.nsys, dtype=torch.int32, device="cuda")
        rr = torch.zeros(B.nsys, dtype=torch.float64, device="cuda")
        res = B.solve(X, to_dev(np.concatenate(rhs)), it, rr, tol=1e-11, mixed=mixed,
                      init_guess_null=not guess)
        assert res.converged == B.nsys
        sols.append(to_host(X))
    assert np.array_equal(*sols)
    for k, (s, b) in enumerate(zip(systems, rhs)):
        x = sols[0][B.sys_row[k]:B.sys_row[k + 1]]
        if k == len(sides) - 1:
            assert np.array_equal(x, x0[B.sys_row[k]:B.sys_row[k + 1]])
            continue
        # the FP64 recurrence's residual drifts by a few roundings an iteration
        assert np.linalg.norm(b - matgen.matvec(*s, x)) <= 2e-11 * np.linalg.norm(b)
        # condition number at most 8.01 / 0.01
        assert np.linalg.norm(x - xs[k]) <= 2e-11 * 801 * np.linalg.norm(xs[k])


def test_chip_irregular_rows(cuda, oracle):
    from seldon_b200 import api
    rng = np.random.default_rng(4)
    systems, rhs = [], []
    for n in (7, 300, 5000):
        m = min(n - 1, 13)
        i = np.repeat(np.arange(n), m)
        j = rng.integers(0, n, i.size)
        keep = (i != j) & (rng.random(i.size) < 0.5)
        key = np.unique(np.concatenate([i[keep] * n + j[keep], j[keep] * n + i[keep]]))
        r, c = key // n, key % n
        d = 1.0 + np.bincount(r, minlength=n)
        key = np.concatenate([key, np.arange(n) * (n + 1)])
        val = np.concatenate([-np.ones(r.size), d])
        at = np.argsort(key)
        r, c, val = key[at] // n, key[at] % n, val[at]
        ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
        systems.append((ptr, c.astype(np.int32), val))
        rhs.append(rng.standard_normal(n))
    B = api.Batch(systems)
    for mixed in (True, False):
        X = to_dev(np.zeros(B.m))
        B.solve(X, to_dev(np.concatenate(rhs)), tol=1e-11, mixed=mixed)
        x = to_host(X)
        for k, (s, b) in enumerate(zip(systems, rhs)):
            xk = x[B.sys_row[k]:B.sys_row[k + 1]]
            assert np.linalg.norm(b - matgen.matvec(*s, xk)) <= 2e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("tuned_mixed", [True, False])
def test_tuned_mode_leaves_the_other_its_plan(cuda, tuned_mixed):
    """A batch tuned in one mode runs the other with its plan, bit for bit."""
    from seldon_b200 import api
    sides = [9, 30, 31, 64, 90]
    systems = [matgen.lap2d(g, shift=0.01) for g in sides]
    b = to_dev(np.random.default_rng(8).uniform(-1, 1, sum(g * g for g in sides)))
    x = [to_dev(np.zeros(b.numel())) for _ in range(2)]
    A, B = api.Batch(systems), api.Batch(systems)
    A.autotune(x[0], b, tol=1e-9, mixed=tuned_mixed)
    B.set_plan(*A.plan(), *A.cluster_plan())
    for v, M in zip(x, (A, B)):
        assert M.solve(v, b, tol=1e-9, mixed=not tuned_mixed).converged == len(sides)
    assert np.array_equal(to_host(x[0]), to_host(x[1]))
