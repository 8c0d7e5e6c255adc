"""Whose errors a host call reports: a ground truth call answers for its own launches
only."""
import numpy as np
import pytest

from distributed_diskann_b200 import datasets as D
from distributed_diskann_b200._lib import DDError
from distributed_diskann_b200.index import GpuIndex

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("dtype", ["u8", "f32"])
def test_ground_truth_leaves_an_earlier_search_error(oracle_mod, dtype):
    import torch

    both = (D.gen_skewed_u8 if dtype == "u8" else D.gen_mixture_f32)(1_100, 32, 8, 5)
    base, q = both[:1_000], np.ascontiguousarray(both[1_000:])
    gi = GpuIndex(base.dtype, "l2", 1_000, 32, 16)
    gi.upload_points(base)
    gi.build(32, 1.2)
    dq = torch.from_numpy(q).cuda()
    L = torch.full((100,), 20, dtype=torch.int32, device="cuda")
    L[3] = 0  # an invalid beam width: reported by check_errors
    ids = torch.zeros((100, 5), dtype=torch.int32, device="cuda")
    ds = torch.zeros((100, 5), device="cuda")
    torch.cuda.synchronize()
    gi.search_device(dq.data_ptr(), 100, dq.stride(0) * dq.element_size(), L.data_ptr(), 20, 5,
                     ids.data_ptr(), ds.data_ptr())
    ti, td = gi.groundtruth(q, 10)
    oi, od = oracle_mod.groundtruth(base, q, 10)
    np.testing.assert_array_equal(ti, oi)
    np.testing.assert_array_equal(td, od)
    with pytest.raises(DDError, match="beam width"):
        gi.check_errors()
    gi.check_errors()
    gi.close()
