"""The persistent sweeps behind SOR and the ILUT apply (csrc/sweep.cuh) at the
sizes where their layout changes: around the block size, one row a level,
rows longer than the entries a thread holds, blocks too large for shared
memory, values that need the full division or look like the fill; bit for
bit against the oracle's sequential loops."""
import numpy as np
import pytest

from seldon_b200 import matgen
from tests.helpers import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(cuda):
    from seldon_b200 import api as a
    return a


def _band(n, offsets, seed, sym):
    """Rows with entries at the given offsets (symmetric pattern), N(0,1) values."""
    rng = np.random.default_rng(seed)
    offs = sorted(set(offsets) | {-o for o in offsets} | {0})
    rows = np.repeat(np.arange(n), len(offs)).reshape(n, -1)
    cols = rows + np.array(offs)
    ok = (cols >= 0) & (cols < n)
    val = rng.standard_normal(cols.shape)
    val[:, offs.index(0)] = 3.0 + 2.0 * len(offs)
    ptr = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int32)
    A = ptr, cols[ok].astype(np.int32), val[ok]
    return matgen.upper(*A) if sym else A


SHAPES = [(1, [1]), (31, [1, 5]), (2047, [1, 40]), (2048, [1]), (2049, [3, 1000]), (4097, [1, 64]),
          (6000, list(range(1, 30))), (30000, [1]), (50000, [7, 300, 20000])]


def _check(api, oracle, A, sym, x0, b, omega, it, t):
    n = A[0].size - 1
    M = api.RowSymSparse(n, *A) if sym else api.RowSparse(n, n, *A)
    X = to_dev(x0)
    api.SOR(M, X, to_dev(b), omega, it, t)
    ref = oracle.sor(*A, x0, b, omega, it, t, sym=sym)
    assert np.array_equal(to_host(X), ref, equal_nan=True)


@pytest.mark.parametrize("n,offsets", SHAPES, ids=[str(s[0]) for s in SHAPES])
@pytest.mark.parametrize("sym", [False, True])
def test_sor_shapes(api, oracle, n, offsets, sym):
    A = _band(n, offsets, n, sym)
    rng = np.random.default_rng(n + 1)
    x0, b = rng.standard_normal(n), rng.standard_normal(n)
    for it, t in ((1, 0), (3, 0), (1, 2), (2, 3), (3, 2), (0, 0)):
        _check(api, oracle, A, sym, x0, b, 1.3, it, t)


@pytest.mark.parametrize("sym", [False, True])
def test_sor_blocks_beyond_shared_memory(api, oracle, sym):
    A = matgen.lap2d(1500)
    A = matgen.upper(*A) if sym else A
    n = A[0].size - 1
    rng = np.random.default_rng(3)
    _check(api, oracle, A, sym, rng.standard_normal(n), rng.standard_normal(n), 1.1, 1, 0)


@pytest.mark.parametrize("sym", [False, True])
def test_sor_special_values(api, oracle, sym):
    ptr, ind, val = _band(3000, [1, 50], 5, False)
    rows = np.repeat(np.arange(3000), np.diff(ptr))
    d = np.flatnonzero(rows == ind)
    val[d[::7]] = 1e-310
    val[d[1::7]] = 1e305
    val[d[2::7]] *= -1.0
    val[d[1500]] = 0.0
    A = matgen.upper(ptr, ind, val) if sym else (ptr, ind, val)
    rng = np.random.default_rng(6)
    x0, b = rng.standard_normal(3000), rng.standard_normal(3000)
    b[::3] = 0.0
    b[1::5] *= 1e-308
    b[2::5] *= 1e300
    b[2900], b[2950] = np.inf, np.nan
    for t in (0, 2, 3):
        _check(api, oracle, A, sym, x0, b, 1.0, 1, t)


@pytest.mark.parametrize("n,offsets", SHAPES, ids=[str(s[0]) for s in SHAPES])
def test_ilu0_shapes(api, oracle, n, offsets):
    A = _band(n, offsets, n + 2, False)
    M = api.IlutPreconditioning()
    M.SetFactorisationType(M.ILU_0)
    H = api.RowSparse(n, n, *A)
    M.FactorizeMatrix(H)
    # the same factor through the host loops of the oracle
    f = _ilu0(*A)
    prow = np.arange(n, dtype=np.int32)
    r = np.random.default_rng(n).standard_normal(n)
    r[n // 2] = np.array([0x7ff4b2005e1d0001], dtype=np.uint64).view(np.float64)[0]
    for trans in (False, True):
        Z = to_dev(np.zeros(n))
        (M.TransSolve if trans else M.Solve)(H, to_dev(r), Z)
        z = oracle.ilut_solve((A[0], A[1], f, prow, prow), r, sym=False, trans=trans)
        assert np.array_equal(to_host(Z), z, equal_nan=True)


def _ilu0(ptr, ind, val):
    """ILU(0) in the row order of the reference, 1 / pivot on the diagonal."""
    ptr, ind, a = ptr.tolist(), ind.tolist(), val.tolist()
    n = len(ptr) - 1
    at = [0] * n
    for i in range(n):
        where = {ind[k]: k for k in range(ptr[i], ptr[i + 1])}
        at[i] = where[i]
        for k in range(ptr[i], at[i]):
            j = ind[k]
            a[k] = a[k] * a[at[j]]
            for q in range(at[j] + 1, ptr[j + 1]):
                if ind[q] in where:
                    a[where[ind[q]]] -= a[k] * a[q]
        a[at[i]] = 1.0 / a[at[i]]
    return np.array(a)


def test_apply_in_a_graph_and_new_values(api, oracle):
    """A captured SSOR apply replays on new data, and later applies read the
    matrix's new values."""
    import ctypes

    import torch
    from seldon_b200 import _lib
    ptr, ind, val = _band(9000, [1, 95], 8, False)
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
    v2 = val * 1.5
    nv = to_dev(v2)
    _lib.check(_lib.load().sb2_csr_set_values(A.handle, ctypes.c_void_p(nv.data_ptr()), 1, None), "set")
    torch.cuda.synchronize()
    S.Solve(A, r, z)
    assert np.array_equal(to_host(z), oracle.sor(ptr, ind, v2, np.zeros(9000), rhs, 1.0, 1, 0))
