"""What a host call refuses, and whose errors it reports: a ground truth call answers for
its own launches only, and query rows closer together than their length are refused at
every size."""
import ctypes as C

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


@pytest.mark.parametrize("nq", [1, 50, 600_000])
def test_query_rows_closer_than_their_length_are_refused(nq):
    base = D.gen_skewed_u8(500, 120, 8, 5)  # 600,000 queries: more than a staging buffer holds
    gi = GpuIndex(base.dtype, "l2", 500, 120, 16)
    gi.upload_points(base)
    gi.build(32, 1.2)
    q = np.zeros((nq, 120), np.uint8)
    Ls = np.full(nq, 20, np.uint32)
    ids, ds = np.zeros((nq, 5), np.uint32), np.zeros((nq, 5), np.float32)
    p = lambda a: C.c_void_p(a.ctypes.data)
    for stride in (119, 60):
        with pytest.raises(DDError):
            gi._ck(gi.lib.dd_search(gi.h, p(q), nq, stride, p(Ls), 5, 1.35, 0, 0, 0, 1, p(ids),
                                    p(ds), None, None))
        with pytest.raises(DDError):
            gi._ck(gi.lib.dd_groundtruth(gi.h, p(q), nq, stride, 5, p(ids), p(ds)))
    gi.search(q, 5, 20)  # the handle goes on
    gi.close()


def test_a_single_query_without_a_stride(oracle_mod):
    base = D.gen_skewed_u8(500, 120, 8, 5)
    gi = GpuIndex(base.dtype, "l2", 500, 120, 16)
    gi.upload_points(base)
    gi.build(32, 1.2)
    q = base[7][None]
    assert q.strides[0] == 0
    oi, od = oracle_mod.groundtruth(base, q, 5)
    ids, ds = gi.groundtruth(q, 5)
    np.testing.assert_array_equal(ids, oi)
    np.testing.assert_array_equal(ds, od)
    np.testing.assert_array_equal(gi.search(q, 5, 20)[0],
                                  gi.search(base[7:8].copy(), 5, 20)[0])
    gi.close()
