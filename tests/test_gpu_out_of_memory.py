"""Calls that run out of device memory fail with an error and leave the handle usable."""
import contextlib

import numpy as np
import pytest

from distributed_diskann_b200 import datasets as D
from distributed_diskann_b200._lib import DDError
from distributed_diskann_b200.index import GpuIndex

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@contextlib.contextmanager
def free_memory(mb):
    """All device memory but about `mb` MB is taken."""
    import torch

    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    assert free > mb * MB
    held = torch.empty(free - mb * MB, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def _rows(gi):
    g = gi.graph()
    g[:, 1:][np.arange(gi.R)[None, :] >= g[:, :1]] = 0
    return g


def test_a_build_that_runs_out_of_memory_leaves_the_handle_usable():
    base = D.gen_mixture_f32(60_000, 16, 60, 3)
    gi = GpuIndex(base.dtype, "l2", 60_000, 16, 64)
    gi.upload_points(base)
    gi.build(64, 1.2, max_build=2_000)
    small = _rows(gi)
    gi.build(64, 1.2)  # rounds of 27,000 points
    large = _rows(gi)
    gi.close()
    gi = GpuIndex(base.dtype, "l2", 60_000, 16, 64)
    gi.upload_points(base)
    gi.build(64, 1.2, max_build=2_000)
    for _ in range(2):
        with free_memory(40):
            with pytest.raises(DDError, match="memory"):
                gi.build(64, 1.2)
    gi.build(64, 1.2, max_build=2_000)
    np.testing.assert_array_equal(_rows(gi), small)
    gi.build(64, 1.2)
    np.testing.assert_array_equal(_rows(gi), large)
    with free_memory(40):
        gi.build(64, 1.2, max_build=2_000)
        gi.build(64, 1.2)  # its scratch is there
    np.testing.assert_array_equal(_rows(gi), large)
    gi.close()
