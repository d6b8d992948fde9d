"""The host's planning of the sweeps (csrc/sweep.cuh, csrc/precond.cu) under the
sanitizers, without a GPU."""
import os
import shutil

import pytest

from tests import test_host_sanitizers as h


@pytest.mark.skipif(not (os.path.exists(h.NVCC) and shutil.which("g++")), reason="needs nvcc and g++")
def test_order_and_items(tmp_path):
    out = h._run([h._driver(str(tmp_path), "fuzz_sweep_plan"), "300"], str(tmp_path))
    h._clean(out)
    assert int(out.split()[1]) > 300
