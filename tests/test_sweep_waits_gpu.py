"""The waits of the persistent sweeps (csrc/sweep.cuh): values that other lanes
and warps of the same block write just before they are read."""
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
