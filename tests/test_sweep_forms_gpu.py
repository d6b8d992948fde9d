"""The forms of the SOR sweeps and the factor's solves (csrc/sweep.cuh): rows that
wait for their values, a launch per level, levels in place; bit for bit
against the oracle's sequential loops, at the sizes where one takes over."""
import numpy as np
import pytest

from seldon_b200 import matgen
from tests.helpers import to_dev, to_host
from tests.test_sweeps_gpu import _band, _check, _ilu0

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(cuda):
    from seldon_b200 import api as a
    return a


def _colored(n, colors, seed, entries=3):
    """Rows of `colors` classes one after the other, joined to rows of other
    classes only: as many levels as classes, at most."""
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(n), entries)
    c = rng.integers(0, n, r.size)
    keep = (r * colors // n) != (c * colors // n)
    r, c = r[keep], c[keep]
    key = np.unique(np.concatenate([r * n + c, c * n + r, np.arange(n) * (n + 1)]))
    r, c = key // n, key % n
    val = rng.standard_normal(key.size)
    val[r == c] = 40.0
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    return ptr, c.astype(np.int32), val


MATRICES = {
    # few levels: rows short and longer than a thread's first entries; below the rows
    # that make a launch pay; one more level than that
    "2 levels": lambda: _colored(9001, 2, 1), "long rows": lambda: _colored(5000, 3, 2, 9),
    "small": lambda: _colored(4095, 2, 3), "16 levels": lambda: _colored(4096, 16, 4),
    "17 levels": lambda: _colored(4096, 17, 5), "diagonal": lambda: _colored(4096, 1, 6),
    # wide rows in narrow levels: one CTA; the same in wider levels
    "band": lambda: _band(3000, list(range(1, 16)), 7, False),
    "wide band": lambda: _band(900, list(range(1, 60)), 8, False),
    "sparse band": lambda: _band(6000, list(range(300, 310)), 9, False),
    # very wide levels: in place, a launch per level
    "1 level": lambda: _colored(200000, 1, 12), "2 wide levels": lambda: _colored(400000, 2, 13),
    "less wide": lambda: _colored(399999, 2, 14),
    "one row": lambda: _band(1, [1], 10, False),
}


@pytest.mark.parametrize("name", list(MATRICES))
@pytest.mark.parametrize("sym", [False, True])
def test_sor_forms(api, oracle, name, sym):
    A = MATRICES[name]()
    n = A[0].size - 1
    A = matgen.upper(*A) if sym else A
    rng = np.random.default_rng(n)
    x0, b = rng.standard_normal(n), rng.standard_normal(n)
    for it, t in ((1, 0), (3, 0), (1, 2), (2, 3), (3, 2), (0, 0)):
        _check(api, oracle, A, sym, x0, b, 1.3, it, t)


@pytest.mark.parametrize("name", list(MATRICES))
@pytest.mark.parametrize("sym", [False, True])
def test_ssor_preconditioner_forms(api, oracle, name, sym):
    """From zero, forward first and backward first, on one handle."""
    A = MATRICES[name]()
    n = A[0].size - 1
    A = matgen.upper(*A) if sym else A
    M = api.RowSymSparse(n, *A) if sym else api.RowSparse(n, n, *A)
    rng = np.random.default_rng(n + 1)
    for order in ((0, 2, 3), (3, 2, 0)):
        S = {0: api.SorPreconditioner(), 2: api.SorPreconditioner(), 3: None}
        S[2].InitUnSymmetricPreconditioning()
        for t in order:
            r = rng.standard_normal(n)
            z = to_dev(np.full(n, 7.0))
            if t == 3:
                S[2].TransSolve(M, to_dev(r), z)
            else:
                S[t].Solve(M, to_dev(r), z)
            assert np.array_equal(to_host(z), oracle.sor(*A, np.zeros(n), r, 1.0, 1, t, sym=sym))


@pytest.mark.parametrize("name", list(MATRICES))
def test_factor_forms(api, oracle, name):
    A = MATRICES[name]()
    n = A[0].size - 1
    M = api.IlutPreconditioning()
    M.SetFactorisationType(M.ILU_0)
    H = api.RowSparse(n, n, *A)
    M.FactorizeMatrix(H)
    f = _ilu0(*A)
    prow = np.arange(n, dtype=np.int32)
    r = np.random.default_rng(n).standard_normal(n)
    for trans in (False, True):
        z = to_dev(np.zeros(n))
        (M.TransSolve if trans else M.Solve)(H, to_dev(r), z)
        assert np.array_equal(to_host(z), oracle.ilut_solve((A[0], A[1], f, prow, prow), r, sym=False, trans=trans))


def test_levels_in_a_graph(api, oracle):
    """A captured apply of launches that overlap replays on new data."""
    import torch
    ptr, ind, val = _colored(9000, 4, 11)
    A = api.RowSparse(9000, 9000, ptr, ind, val)
    S = api.SorPreconditioner()
    r, z = to_dev(np.ones(9000)), to_dev(np.zeros(9000))
    S.Solve(A, r, z)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        S.Solve(A, r, z)
    rhs = np.random.default_rng(9).standard_normal(9000)
    r.copy_(to_dev(rhs))
    g.replay()
    assert np.array_equal(to_host(z), oracle.sor(ptr, ind, val, np.zeros(9000), rhs, 1.0, 1, 0))
