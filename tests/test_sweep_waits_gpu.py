"""The waits of the persistent sweeps (csrc/sweep.cuh): values that other lanes
and warps of the same block write just before they are read, a wait that runs
out (the plan is made to hold a value that never comes, and each wait ends by
the clock, a second or two later) and a row that takes longer than the limit."""
import numpy as np
import pytest

from tests.helpers import to_dev, to_host

pytestmark = pytest.mark.gpu


def _layered(layers, width, seed):
    """Rows in layers of `width`, each reading rows of the layer before and of
    the layer behind at random, so that the levels of both sweeps are the
    layers and a row reads what any lane of any warp wrote a step before."""
    rng = np.random.default_rng(seed)
    n = layers * width
    rows, cols = [np.arange(n)], [np.arange(n)]
    for a in range(layers - 1):
        r = np.repeat(np.arange((a + 1) * width, (a + 2) * width), 3)
        c = a * width + rng.integers(0, width, r.size)
        rows += [r, c]
        cols += [c, r]
    key = np.unique(np.concatenate(rows) * n + np.concatenate(cols))
    r, c = key // n, key % n
    val = rng.standard_normal(key.size)
    val[r == c] = 12.0
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    return ptr, c.astype(np.int32), val


@pytest.mark.parametrize("layers,width", [(60, 33), (20, 100), (4, 512), (200, 65)])
def test_values_of_other_lanes_in_the_block(cuda, oracle, layers, width):
    from seldon_b200 import api
    ptr, ind, val = _layered(layers, width, width)
    n = ptr.size - 1
    A = api.RowSparse(n, n, ptr, ind, val)
    rng = np.random.default_rng(n)
    S = api.SorPreconditioner()
    for _ in range(20):
        b = rng.standard_normal(n)
        z = to_dev(np.zeros(n))
        S.Solve(A, to_dev(b), z)
        assert np.array_equal(to_host(z), oracle.sor(ptr, ind, val, np.zeros(n), b, 1.0, 1, 0))


@pytest.fixture
def short_limit(cuda):
    """The sweeps' wait limit at its floor of a second."""
    from seldon_b200 import _lib
    L = _lib.load()
    old = L.sb2_set_wait_limit_us(1)
    yield L
    L.sb2_set_wait_limit_us(old)


@pytest.fixture(scope="module")
def breaker(cuda):
    """tests/cuda/sweep_wait.cu: points an entry of a sweep's plan elsewhere."""
    import ctypes
    import os
    import subprocess
    here = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cuda")
    subprocess.run(["make", "-C", here, "sweep_wait.so"], check=True, capture_output=True)
    lib = ctypes.CDLL(os.path.join(here, "sweep_wait.so"))

    def point(handle, sweep, entry, at):
        old = ctypes.c_int()
        assert lib.break_sweep(handle, sweep, entry, at, ctypes.byref(old)) == 0
        return old.value
    return point


N = 6000  # three blocks of 2000 rows, a chain through all of them


def _chain_factor(api):
    """L and U of one off-diagonal each (Seldon's layout: L, 1/U(i,i), U)."""
    i = np.arange(N)
    rows = np.concatenate([i[1:], i, i[:-1]])
    cols = np.concatenate([i[1:] - 1, i, i[:-1] + 1])
    vals = np.concatenate([np.full(N - 1, -0.3), np.full(N, 0.8), np.full(N - 1, -0.2)])
    at = np.lexsort((cols, rows))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=N))]).astype(np.int32)
    f = ptr, cols[at].astype(np.int32), vals[at]
    M = api.IlutPreconditioning()
    M.SetFactor(*f, i.astype(np.int32), i.astype(np.int32))
    return M, (*f, i.astype(np.int32), i.astype(np.int32))


def _tridiagonal(api):
    i = np.arange(N)
    rows = np.concatenate([i[1:], i, i[:-1]])
    cols = np.concatenate([i[1:] - 1, i, i[:-1] + 1])
    vals = np.concatenate([np.full(N - 1, -1.0), np.full(N, 4.0), np.full(N - 1, -1.0)])
    at = np.lexsort((cols, rows))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=N))]).astype(np.int32)
    return api.RowSparse(N, N, ptr, cols[at].astype(np.int32), vals[at])


def test_apply_whose_wait_runs_out(short_limit, breaker, oracle):
    """Two rows of a plan wait for one another: the apply ends by the clock, the
    rows not reached are NaN, the status call tells once, a solver that comes
    after is not blamed, and the plan mended applies as before."""
    import ctypes

    from seldon_b200 import _lib, api
    L = short_limit
    A = _tridiagonal(api)
    M, f = _chain_factor(api)
    h = M.handle_for(A)
    r = np.random.default_rng(1).standard_normal(N)
    good = oracle.ilut_solve(f, r, sym=False, trans=False)

    def status():
        v = ctypes.c_int(-1)
        _lib.check(L.sb2_precond_status(h, None, ctypes.byref(v)), "status")
        return v.value

    def apply():
        z = to_dev(np.full(N, 7.0))
        M.Solve(A, to_dev(r), z)
        return to_host(z)

    def cg(iters):
        x, it = to_dev(np.zeros(N)), api.Iteration(iters, 1e-10)
        it.HideMessages()
        api.Cg(A, x, to_dev(r), M, it)
        return to_host(x)

    assert np.array_equal(apply(), good) and status() == 0
    x = cg(3)
    # L sweep: row 1 waits for the last row, which waits for it through the chain
    was = breaker(h, 0, 0, N - 1)
    assert was == 0
    z = apply()
    assert np.isnan(z).all()
    assert status() == 1 and status() == 0
    apply()
    with pytest.raises(_lib.SeldonB200Error) as err:
        cg(1)
    assert err.value.status == _lib.SB2_ERR_TIMEOUT
    breaker(h, 0, 0, was)
    # the direct apply's word is still set, and is not the solver's
    assert np.array_equal(cg(3), x)
    assert status() == 1 and status() == 0
    # U sweep: row 3999 waits for row 1999 and so for itself; rows 4000.. are done
    was = breaker(h, 1, 2000, 0)
    z = apply()
    assert np.isnan(z[:4000]).all() and np.array_equal(z[4000:], good[4000:])
    assert status() == 1
    breaker(h, 1, 2000, was)
    assert np.array_equal(apply(), good) and status() == 0


def test_long_row_is_progress(short_limit, oracle):
    """A row whose sum takes one lane longer than the wait limit: the row that
    waits for it goes on waiting."""
    from seldon_b200 import api
    n, chain = 6_000_000, 420  # (a chain of rows: with few levels each would be a launch)
    long = n - 2
    one = np.arange(long)
    rows = np.concatenate([one, one[1:chain], np.full(long + 1, long), [n - 1, n - 1]])
    cols = np.concatenate([one, one[:chain - 1], np.arange(long + 1), [long, n - 1]])
    ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    at = np.lexsort((cols, rows))
    ind = cols[at].astype(np.int32)
    val = np.where(rows[at] == ind, 2.0, np.where(rows[at] == long, 1e-7, 0.5))
    rng = np.random.default_rng(2)
    x0, b = rng.standard_normal(n), rng.standard_normal(n)
    x = to_dev(x0)
    api.SOR(api.RowSparse(n, n, ptr, ind, val), x, to_dev(b), 1.0, 1, 2)
    assert np.array_equal(to_host(x), oracle.sor(ptr, ind, val, x0, b, 1.0, 1, 2, sym=False))
