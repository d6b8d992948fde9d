"""The forms of the COO assembly (csrc/assemble.cu) at the sizes where one takes
over from another: triplets in order, buckets of rows, the row scatter; each
against a stable sort of the triplets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(r, c, v, m, sym):
    if sym:
        keep = r <= c
        r, c, v = r[keep], c[keep], v[keep]
    at = np.lexsort((np.arange(r.size), c, r))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m))]).astype(np.int32)
    return ptr, c[at].astype(np.int32), v[at]


def _check(r, c, v, index, m0, sym):
    import torch
    from seldon_b200 import api
    m, n, ptr, ind, val = api.ConvertMatrix_from_Coordinates(
        torch.as_tensor((r + index).astype(np.int32)).cuda(), torch.as_tensor((c + index).astype(np.int32)).cuda(),
        torch.as_tensor(v).cuda(), index, m0, 0, sym)
    want_m = int(r.max()) + 1 if sym else max(int(r.max()) + 1, m0)
    assert m == want_m
    p, i, x = _reference(r, c, v, m, sym)
    assert np.array_equal(ptr.cpu().numpy(), p)
    assert np.array_equal(ind.cpu().numpy(), i)
    assert np.array_equal(val.cpu().numpy(), x)


# (triplets, rows, columns, longest row's share): tiles are 8192 triplets, a
# bucket holds 5376 entries and 4096 rows, a row of 48 is the last ranked one
CASES = [(1, 1, 1, 0.0), (5, 3, 7, 0.0), (8192, 100, 1000, 0.0), (8193, 5000, 5000, 0.0),
         (40000, 3, 100000, 0.0), (60000, 1200, 300, 0.0), (200000, 100000, 50, 0.0),
         (20000, 30000000, 10, 0.0), (300000, 4096, 2000000000, 0.0), (100000, 5000, 5000, 0.2),
         (1000000, 4097, 20000, 0.0), (500000, 10000, 9000, 0.004)]


@pytest.mark.parametrize("nnz,m,n,share", CASES, ids=[f"{c[0]}-{c[1]}-{c[3]}" for c in CASES])
@pytest.mark.parametrize("order", ["random", "sorted", "nearly"])
@pytest.mark.parametrize("sym", [False, True])
def test_forms(cuda, nnz, m, n, share, order, sym):
    rng = np.random.default_rng(nnz + m)
    r = rng.integers(0, m, nnz).astype(np.int64)
    c = rng.integers(0, min(n, m) if sym else n, nnz).astype(np.int64)
    r[rng.random(nnz) < share] = m // 2
    c[rng.random(nnz) < 0.1] = c[0]  # duplicates
    if sym and order != "random":  # nothing to drop: the copying form
        r, c = np.minimum(r, c), np.maximum(r, c)
    if order != "random":
        at = np.lexsort((c, r))
        r, c = r[at], c[at]
    if order == "nearly" and nnz > 1:
        r[[nnz // 3, -1]] = r[[-1, nnz // 3]]
    v = rng.standard_normal(nnz)
    _check(r, c, v, 1 if nnz % 2 else 0, m + 5, sym)
