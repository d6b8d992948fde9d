"""Cg, BiCgStab and Gmres with their vectors in shared memory (csrc/resident.cuh)
against the oracle, at the sizes where the layout changes: rows that fill no
whole quad or slice, one and several slices a CTA, the matrix on chip and not,
rows of differing length, an initial guess, a right-hand side and a solution
that start off a 16-byte boundary."""
import numpy as np
import pytest

from seldon_b200 import matgen
from tests.helpers import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(cuda):
    from seldon_b200 import api as a
    return a


def _ragged(n, seed, sym):
    """Diagonally dominant rows of 1 to 9 entries (kept in row order)."""
    rng = np.random.default_rng(seed)
    offs = np.array([1, 2, 37, 300])
    r = np.repeat(np.arange(n), offs.size)
    c = r + np.tile(offs, n)
    keep = (c < n) & (rng.random(r.size) < 0.6)
    r, c = r[keep], c[keep]
    v = rng.uniform(-1, 0, r.size)
    w = v if sym else rng.uniform(-1, 0, r.size)
    rows = np.concatenate([r, c, np.arange(n)])
    cols = np.concatenate([c, r, np.arange(n)])
    vals = np.concatenate([v, w, np.zeros(n)])
    vals[-n:] = 0.5 + np.bincount(rows, weights=np.abs(vals), minlength=n)
    at = np.lexsort((cols, rows))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return ptr, cols[at].astype(np.int32), vals[at]


# (solver, matrix, rows the operator has, restart, most iterations)
CASES = [
    ("cg", "lap", 301 * 301, 10, 5000),
    ("cg", "ragged_sym", 131073, 10, 500),
    ("cg", "ragged_sym", 200002, 10, 500),
    ("bicgstab", "conv", 33 ** 3, 10, 500),
    ("bicgstab", "ragged", 19001, 10, 500),
    ("bicgstab", "ragged", 127, 10, 500),
    ("gmres", "conv", 33 ** 3, 7, 1000),
    ("gmres", "ragged", 147 * 128 + 3, 30, 500),
    ("gmres", "ragged", 150 * 128 + 1, 1, 500),
    ("gmres", "ragged", 400001, 12, 100),
    ("gmres", "conv", 71 ** 3, 10, 40),
]


def _matrix(name, n):
    if name == "lap":
        return matgen.lap2d(round(n ** 0.5))
    if name == "conv":
        return matgen.convdiff3d(round(n ** (1 / 3)))
    return _ragged(n, n, name == "ragged_sym")


@pytest.mark.parametrize("which,name,n,restart,most", CASES, ids=[f"{c[0]}-{c[1]}-{c[2]}" for c in CASES])
@pytest.mark.parametrize("jacobi", [False, True])
@pytest.mark.parametrize("guess", [False, True])
def test_resident_vs_oracle(api, oracle, which, name, n, restart, most, jacobi, guess):
    import torch
    ptr, ind, val = _matrix(name, n)
    assert ptr.size - 1 == n
    rng = np.random.default_rng(n + restart)
    b = matgen.matvec(ptr, ind, val, rng.uniform(-1, 1, n))
    x0 = rng.uniform(-1, 1, n) if guess else None
    A = api.RowSparse(n, n, ptr, ind, val)
    # one entry into a buffer: 8-byte aligned only
    X = torch.zeros(n + 1, dtype=torch.float64, device="cuda")[1:]
    B = torch.zeros(n + 1, dtype=torch.float64, device="cuda")[1:]
    B.copy_(to_dev(b))
    if guess:
        X.copy_(to_dev(x0))
    it = api.Iteration(most, 1e-10)
    it.SetRestart(restart)
    it.HideMessages()
    it.SetInitGuess(not guess)
    M = api.JacobiPreconditioner() if jacobi else api.Preconditioner_Base()
    f = {"cg": api.Cg, "bicgstab": api.BiCgStab, "gmres": api.Gmres}[which]
    code = f(A, X, B, M, it)
    xo, co, no, _, _ = oracle.solve(which, ptr, ind, val, b, x0=x0, precond=1 if jacobi else 0, tol=1e-10,
                                    max_iter=most, restart=restart)
    assert code == co
    assert abs(it.GetNumberIteration() - no) <= max(2, no // 20)
    # the residuals agree to 1e-10 of ||b||; these operators' condition
    # numbers stay below 1e5 (301^2 Laplacian: 4e4)
    x = to_host(X)
    assert np.linalg.norm(x - xo) <= 1e-5 * np.linalg.norm(xo) * (1.0 if co == 0 else 10.0)
    r = b - matgen.matvec(ptr, ind, val, x)
    ro = b - matgen.matvec(ptr, ind, val, xo)
    if co == 0:
        assert np.linalg.norm(r) <= 2e-10 * np.linalg.norm(b) + 2 * np.linalg.norm(ro)


@pytest.mark.parametrize("long_row", [False, True])
@pytest.mark.parametrize("restart,taken", [(140, True), (141, False), (200, False), (1000, False)])
def test_restarts_taken(api, long_row, restart, taken):
    """Gmres takes the same restarts whichever of its kernels a matrix runs on
    (a row of more than 32 entries keeps it off the chip)."""
    import torch
    from seldon_b200 import _lib
    n = 3000
    ptr, ind, val = _ragged(n, 5, False)
    if long_row:
        k = ptr[1]
        cols = np.union1d(ind[:k], np.arange(0, 400, 8)).astype(np.int32)
        row0 = np.full(cols.size, 1e-3)
        row0[0] = 2.0
        ind = np.concatenate([cols, ind[k:]])
        val = np.concatenate([row0, val[k:]])
        ptr = np.concatenate([[0], ptr[1:] + cols.size - k]).astype(np.int32)
    A = api.RowSparse(n, n, ptr, ind, val)
    b = to_dev(np.random.default_rng(6).standard_normal(n))
    x = torch.zeros_like(b)
    it = api.Iteration(2, 1e-10)
    it.SetRestart(restart)
    it.HideMessages()
    if taken:
        api.Gmres(A, x, b, api.Preconditioner_Base(), it)
        # (a cycle runs to its restart or the tolerance, whatever max_iter is)
        assert 2 <= it.GetNumberIteration() <= restart
    else:
        with pytest.raises(_lib.SeldonB200Error) as err:
            api.Gmres(A, x, b, api.Preconditioner_Base(), it)
        assert err.value.status == _lib.SB2_ERR_NOT_SUPPORTED


@pytest.mark.parametrize("n", [148 * 8192, 148 * 8192 + 1])
@pytest.mark.parametrize("restart", [3, 4, 17, 18])
def test_gmres_where_the_forms_change(api, oracle, n, restart):
    """Up to 8192 rows a CTA and one more, at the restarts where the fused kernel
    hands over."""
    test_resident_vs_oracle(api, oracle, "gmres", "ragged", n, restart, 20, True, False)


@pytest.mark.parametrize("which,name,n", [("cg", "lap", 301 * 301), ("bicgstab", "ragged_sym", 19001),
                                          ("gmres", "ragged_sym", 70001)])
@pytest.mark.parametrize("jacobi", [False, True])
def test_resident_symmetric_storage(api, oracle, which, name, n, jacobi):
    """The expanded rows of symmetric storage, against the oracle's general ones."""
    import torch
    ptr, ind, val = _matrix(name, n)
    b = matgen.matvec(ptr, ind, val, np.random.default_rng(n).uniform(-1, 1, n))
    A = api.RowSymSparse(n, *matgen.upper(ptr, ind, val))
    X = torch.zeros(n, dtype=torch.float64, device="cuda")
    it = api.Iteration(5000, 1e-10)
    it.SetRestart(20)
    it.HideMessages()
    M = api.JacobiPreconditioner() if jacobi else api.Preconditioner_Base()
    code = {"cg": api.Cg, "bicgstab": api.BiCgStab, "gmres": api.Gmres}[which](A, X, to_dev(b), M, it)
    xo, co, no, _, _ = oracle.solve(which, ptr, ind, val, b, precond=1 if jacobi else 0, tol=1e-10,
                                    max_iter=5000, restart=20)
    assert code == co == 0
    assert abs(it.GetNumberIteration() - no) <= max(2, no // 20)
    assert np.linalg.norm(to_host(X) - xo) <= 1e-5 * np.linalg.norm(xo)
