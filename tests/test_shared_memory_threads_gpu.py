"""Calls from several host threads, each on its own stream and matrix, whose
kernels are the same and take different amounts of shared memory: no call may
be refused because another one's amount is smaller."""
import threading

import numpy as np
import pytest

from seldon_b200 import matgen
from tests.helpers import to_dev, to_host

pytestmark = pytest.mark.gpu


def _solver(api, torch, name, size, stream):
    """One small solve of a system of the given size: (call, its solution)."""
    sp = stream.cuda_stream
    rng = np.random.default_rng(size)
    it = api.Iteration(3, 1e-10)
    it.HideMessages()
    if name == "batch":
        systems = [matgen.lap2d(size, shift=0.01)] * 3
        B = api.Batch(systems)
        x, b = to_dev(np.zeros(B.m)), to_dev(rng.standard_normal(B.m))
        d, r = torch.zeros(3, dtype=torch.int32, device="cuda"), to_dev(np.zeros(3))
        return lambda: B.solve(x, b, d, r, summary=False, max_iter=3, tol=1e-10, stream=sp), x, B
    n = size * size
    A = api.RowSparse(n, n, *matgen.lap2d(size))
    x, b = to_dev(np.zeros(n)), to_dev(rng.standard_normal(n))

    if name == "sor":
        S = api.SorPreconditioner()
        return lambda: S.Solve(A, b, x, stream=sp), x, (A, S)

    def call():
        if name == "cgs2":
            it.SetRestart(1 + size % 20)
            api.Gmres(A, x, b, api.Preconditioner_Base(), it, stream=sp, orthogonalization="cgs2")
        else:
            it.SetRestart(size)
            {"cg": api.Cg, "gmres": api.Gmres}[name](A, x, b, api.Preconditioner_Base(), it, stream=sp)
    return call, x, A


# sides of the systems: of one cluster, of the batch's largest, of Gmres (whose
# restart follows the side), of the sweeps' blocks; resident: of the whole chip
CASES = {"cg": [40, 60, 100, 140], "batch": [50, 70, 90, 140], "cgs2": [41, 45, 50, 59],
         "sor": [700, 1000, 1200, 1400]}


@pytest.mark.parametrize("name", list(CASES) + ["resident"])
def test_same_kernel_other_sizes(cuda, name):
    import torch
    from seldon_b200 import api
    sizes = CASES.get(name, [300, 350, 400, 450])
    which = {"resident": "cg"}.get(name, name)
    streams = [torch.cuda.Stream() for _ in sizes]
    work = [_solver(api, torch, which, g, s) for g, s in zip(sizes, streams)]
    torch.cuda.synchronize()
    want = []
    for call, x, _ in work:
        call()
        torch.cuda.synchronize()
        want.append(to_host(x).copy())
    start, err = threading.Barrier(len(sizes)), []

    def run(k):
        try:
            start.wait()
            for _ in range(60 if name == "sor" else 400):
                work[k][0]()
        except Exception as e:  # reported below, on the main thread
            err.append(e)

    ts = [threading.Thread(target=run, args=(k,)) for k in range(len(sizes))]
    for t in ts:
        t.start()
    for t in ts:
        t.join(timeout=120)
    assert not any(t.is_alive() for t in ts)
    assert not err, err
    torch.cuda.synchronize()
    for (_, x, _), w in zip(work, want):
        assert np.array_equal(to_host(x), w)
