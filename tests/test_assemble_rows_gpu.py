"""The COO assembly (csrc/assemble.cu) where rows are missing: triplets in order
with runs of empty rows before, between and behind them, around the length that
one thread fills; and where rows are long, around the lengths that buckets rank,
sort and leave to the row form."""
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


@pytest.mark.parametrize("length", [47, 49, 65, 81, 447, 448, 449, 513, 900])
@pytest.mark.parametrize("sym", [False, True])
def test_rows_of_a_length(cuda, length, sym):
    """Rows of this many entries and one of each neighbouring length, shuffled."""
    rng = np.random.default_rng(length)
    m = 300
    lens = np.full(m, length)
    lens[[3, 100]] = length - 1
    lens[[7, 200]] = length + 1
    lens[50] = 0
    r = np.repeat(np.arange(m), lens)
    c = rng.integers(0, 40 if length % 2 else 100000, r.size)
    if sym:
        c = c % m
    at = rng.permutation(r.size)
    _check(r[at], c[at], rng.standard_normal(r.size), 0, m, sym)


@pytest.mark.parametrize("mean", [400, 430, 1100])
def test_many_triplets_in_long_rows(cuda, mean):
    """4M triplets and more, where the mean row decides the form."""
    rng = np.random.default_rng(mean)
    nnz = 4_100_000
    m = nnz // mean
    _check(rng.integers(0, m, nnz), rng.integers(0, m, nnz), rng.standard_normal(nnz), 0, m, False)


def _starved():
    import torch
    from seldon_b200 import api
    nnz, m = 18 << 20, 1 << 22  # 4096 buckets of 4608 entries
    gen = torch.Generator(device="cuda").manual_seed(5)
    row = torch.randint(0, m, (nnz,), device="cuda", dtype=torch.int32, generator=gen)
    col = torch.randint(0, 1000, (nnz,), device="cuda", dtype=torch.int32, generator=gen)
    val = torch.ones(nnz, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # outputs of 12 bytes a triplet and a row's 4 (232 MB), then 288 MB of scratch
    # or 144 MB and two arrays of a row's 4 (176 MB)
    free = torch.cuda.mem_get_info()[0]
    spare = (232 + 232) << 20
    assert free > spare
    full = torch.empty(free - spare, dtype=torch.uint8, device="cuda")
    try:
        M, N, ptr, ind, v = api.ConvertMatrix_from_Coordinates(row, col, val, 0, m, 0, False)
    finally:
        del full
        torch.cuda.empty_cache()
    count = torch.bincount(row, minlength=m)
    assert M == m and torch.equal(torch.diff(ptr).long(), count)
    assert int(ind.long().sum()) == int(col.long().sum()) and bool((v == 1.0).all())
    # columns in order within each row
    same = torch.ones(nnz - 1, dtype=torch.bool, device="cuda")
    ends = ptr[1:-1].long()
    same[ends[(ends > 0) & (ends < nnz)] - 1] = False
    assert bool((ind[1:] >= ind[:-1])[same].all())


def test_scratch_that_does_not_fit(cuda):
    """The bucket form's scratch is 16 bytes a triplet, the row form's 8: with
    room for the second only the call still succeeds.  (A process of its own: no
    memory that earlier calls left in the library's pool.)"""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = "from tests.test_assemble_rows_gpu import _starved; _starved(); print('starved: done')"
    p = subprocess.run([sys.executable, "-c", run], cwd=root, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and "starved: done" in p.stdout, p.stderr[-3000:]
