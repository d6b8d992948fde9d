"""The size classes of the batched solve with vectors in shared memory
(csrc/batch.cu): a launch each, overlapping on one stream."""
import numpy as np
import pytest

from tests.helpers import to_dev, to_host

pytestmark = pytest.mark.gpu


def _chain(n, shift=0.5):
    """1D Laplacian of n rows, shifted: condition number below (4 + shift) / shift."""
    i = np.arange(n)
    rows = np.concatenate([i[1:], i, i[:-1]])
    cols = np.concatenate([i[1:] - 1, i, i[:-1] + 1])
    vals = np.concatenate([np.full(n - 1, -1.0), np.full(n, 2.0 + shift), np.full(n - 1, -1.0)])
    at = np.lexsort((cols, rows))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return ptr, cols[at].astype(np.int32), vals[at]


# rows of the systems: around the classes' limits, one class empty, one system,
# more small systems than fit at once behind a large one
BATCHES = {"limits": [511, 512, 513, 2047, 2048, 2049, 1, 14000], "no middle": [3000, 100, 7],
           "no large": [600, 2048, 5, 512], "small": [1, 2, 512], "one": [2049],
           "behind": [9000] + [64] * 5000 + [700] * 900}


@pytest.mark.parametrize("name", list(BATCHES))
@pytest.mark.parametrize("mixed", [True, False])
def test_classes(cuda, name, mixed):
    import torch

    from seldon_b200 import api
    rng = np.random.default_rng(len(name))
    sizes = np.array(BATCHES[name])[rng.permutation(len(BATCHES[name]))]
    made = {int(n): _chain(int(n)) for n in set(sizes)}
    B = api.Batch([made[int(n)] for n in sizes])
    want = rng.uniform(-1, 1, B.m)
    b = np.concatenate([(2.5 * x - np.append(x[1:], 0.0) - np.append(0.0, x[:-1]))
                        for x in np.split(want, B.sys_row[1:-1])])
    bd = to_dev(b)
    it = torch.zeros(B.nsys, dtype=torch.int32, device="cuda")
    rr = torch.zeros(B.nsys, dtype=torch.float64, device="cuda")
    x = to_dev(np.zeros(B.m))
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(3):  # what follows on the stream follows every class
            x.fill_(np.nan)
            it.fill_(-1)
            B.solve(x, bd, it, rr, summary=False, tol=1e-11, mixed=mixed, stream=side.cuda_stream)
            y, n = x.clone(), it.clone()
    side.synchronize()
    assert torch.equal(x, y) and torch.equal(it, n)
    assert int(it.min()) >= 1 and float(rr.max()) < 1e-11
    # ||e|| <= cond ||r|| / ||A||, system by system (the FP64 recurrence's residual
    # drifts by a few roundings an iteration)
    for k, (u, w) in enumerate(zip(np.split(to_host(x), B.sys_row[1:-1]), np.split(want, B.sys_row[1:-1]))):
        assert np.linalg.norm(u - w) <= 9 * 2e-11 * 4.5 * np.linalg.norm(w), (k, sizes[k])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        B.solve(x, bd, it, rr, summary=False, tol=1e-11, mixed=mixed)
    x.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(x, y) and torch.equal(it, n)


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("per_sm,planned", [(3, False), (4, True)])
def test_systems_that_do_not_fit(cuda, mixed, per_sm, planned):
    """With four systems an SM too large for shared memory an untuned batch runs
    the default plan (the same bits), with fewer it does not."""
    import torch

    from seldon_b200 import api
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 28673 if mixed else 14337  # one row more than 224 KB hold twice
    assert 2 * n * (4 if mixed else 8) > 224 * 1024
    rng = np.random.default_rng(per_sm)
    big, fits = _chain(n), _chain(n - 1)
    systems = [big] * (per_sm * sms) + [fits] * 5
    xs = []
    b = to_dev(rng.uniform(-1, 1, per_sm * sms * n + 5 * (n - 1)))
    for plan in (False, True):
        B = api.Batch(systems)
        if plan:
            B.set_plan(256, 0)
        x = to_dev(np.zeros(B.m))
        it = torch.zeros(B.nsys, dtype=torch.int32, device="cuda")
        rr = torch.zeros(B.nsys, dtype=torch.float64, device="cuda")
        B.solve(x, b, it, rr, summary=False, tol=1e-30, max_iter=20, mixed=mixed)
        xs.append(x)
        B.close()
    assert torch.equal(*xs) == planned
    assert float((xs[0] - xs[1]).norm()) <= 1e-5 * float(xs[1].norm())


def test_tuning_is_kept_by_what_fits(cuda):
    """A batch with the sizes of a tuned one and other rows is timed itself; one
    with the same rows takes the tuned plan without timing."""
    from seldon_b200 import api
    rng = np.random.default_rng(3)
    n = 1500

    def banded(k):
        i = np.repeat(np.arange(n), 2 * k + 1)
        j = i + np.tile(np.arange(-k, k + 1), n)
        ok = (j >= 0) & (j < n)
        i, j = i[ok], j[ok]
        ptr = np.concatenate([[0], np.cumsum(np.bincount(i, minlength=n))]).astype(np.int32)
        return ptr, j.astype(np.int32), np.where(i == j, 4.0 * k, -1.0)

    b = to_dev(rng.uniform(-1, 1, 40 * n))

    def timed(k):
        B = api.Batch([banded(k)] * 40)
        x = to_dev(np.full(B.m, 7.0))
        B.autotune(x, b, tol=1e-6)
        return bool((x != 7.0).any())

    assert timed(2) and not timed(2)
    assert timed(13) and not timed(13)
