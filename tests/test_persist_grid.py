"""The grid of the persistent solvers follows a matrix's entries, not its rows
alone; and a solve whose long rows are dealt to groups of threads."""
import os
import shutil

import numpy as np
import pytest

from tests.helpers import to_dev, to_host


def test_grid_covers_the_entries(tmp_path):
    from tests import test_host_sanitizers as h
    if not (os.path.exists(h.NVCC) and shutil.which("g++")):
        pytest.skip("needs nvcc and g++")
    # (rows, entries a row): CTAs of 1024 threads at least
    cases = {(8192, 300): 148, (4096, 1000): 148, (20000, 81): 148, (27000, 27): 80, (30000, 5): 30,
             (1000, 3): 1, (1, 1): 1, (2000000, 7): 148}
    exe = h._driver(str(tmp_path), "grid_rule")
    got = h._run([exe] + [str(v) for c in cases for v in c], str(tmp_path)).split()
    for (c, least), n in zip(cases.items(), map(int, got)):
        assert least <= n <= 148, (c, n)


def _long_rows(n, count, length, seed):
    """5-entry rows, and `count` of about `length` entries; off the diagonal they sum to less than 1."""
    rng = np.random.default_rng(seed)
    at = rng.choice(n, count, replace=False)
    rows = np.concatenate([np.repeat(np.arange(n), 4)] + [np.full(length, r) for r in at])
    cols = np.concatenate([rng.integers(0, n, 4 * n)] + [rng.choice(n, length, replace=False) for _ in at])
    off = rows != cols
    key = np.unique(np.concatenate([rows[off] * n + cols[off], np.arange(n) * (n + 1)]))
    r, c = key // n, key % n
    deg = np.bincount(r, minlength=n)
    val = rng.uniform(-1, 1, key.size) / deg[r]
    val[r == c] = 2.0
    ptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    return ptr, c.astype(np.int32), val


# rows of the CTA bin (more than 1024 entries): none, fewer than CTAs, more than
# CTAs (groups of 256 threads), lengths around the groups' strides
@pytest.mark.gpu
@pytest.mark.parametrize("n,count,length", [(3000, 0, 0), (3000, 1, 2900), (3000, 30, 1100), (6000, 400, 1029),
                                            (6000, 200, 2048), (9000, 700, 1500)])
@pytest.mark.parametrize("which", ["bicgstab", "cgs", "lsqr"])
def test_long_rows_by_groups(cuda, oracle, n, count, length, which):
    from seldon_b200 import api
    ptr, ind, val = _long_rows(n, count, length, n + count)
    b = np.random.default_rng(count).standard_normal(n)
    x, it = to_dev(np.zeros(n)), api.Iteration(200, 1e-11)
    it.HideMessages()
    f = {"bicgstab": api.BiCgStab, "cgs": api.Cgs, "lsqr": api.Lsqr}[which]
    code = f(api.RowSparse(n, n, ptr, ind, val), x, to_dev(b), api.JacobiPreconditioner(), it)
    xo, co, no, _, _ = oracle.solve(which, ptr, ind, val, b, precond=1, tol=1e-11, max_iter=200)
    assert code == co == 0
    assert abs(it.GetNumberIteration() - no) <= 2
    # both residuals are below 1e-11 ||b|| and the eigenvalues within 1 of 2
    assert np.linalg.norm(to_host(x) - xo) <= 4e-11 * np.linalg.norm(b)
