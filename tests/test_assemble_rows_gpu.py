"""The COO assembly (csrc/assemble.cu) where rows are missing: triplets in order
with runs of empty rows before, between and behind them, around the length that
one thread fills."""
import numpy as np
import pytest

from tests.test_assemble_forms_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap", [1, 2047, 2048, 2049, 100000, 200000])
@pytest.mark.parametrize("where", ["first", "between", "last", "size"])
@pytest.mark.parametrize("index", [0, 1])
def test_runs_of_empty_rows(cuda, gap, where, index):
    rng = np.random.default_rng(gap)
    nnz = 30000
    r = np.sort(rng.integers(0, 50, nnz))
    if where == "first":
        r += gap
    elif where == "between":
        r[nnz // 2:] += gap
    elif where == "last":
        r[-1] += gap
    c = rng.integers(0, 1000, nnz)
    at = np.lexsort((c, r))
    m0 = int(r.max()) + (gap if where == "size" else 1)
    _check(r[at], c[at], rng.standard_normal(nnz), index, m0, False)


def test_one_long_run_takes_no_longer_than_a_search(cuda):
    """16M empty rows before the last triplet: the call's device time is that of
    moving the arrays, not of one thread's stores (56 ms)."""
    import torch
    from seldon_b200 import api
    nnz = 4_000_000
    row = torch.arange(nnz, device="cuda", dtype=torch.int32) // 4000
    row[-1] = 15_999_999
    col, val = torch.zeros_like(row), torch.ones(nnz, dtype=torch.float64, device="cuda")
    best = 1e9
    for _ in range(4):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        m, n, ptr, ind, v = api.ConvertMatrix_from_Coordinates(row, col, val, 0, 0, 0, False)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    assert m == 16_000_000 and int(ptr[-1]) == nnz and int(ptr[-2]) == nnz - 1 and int(ptr[1001]) == nnz - 1
    assert best < 10.0
