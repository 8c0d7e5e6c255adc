"""The sharded build's integer searches read every row's norm from an array that is made
once a build, not once a round, and again when the points change."""
import numpy as np
import pytest

from distributed_diskann_b200 import datasets as D
from distributed_diskann_b200.index import GpuIndex
from distributed_diskann_b200.sharded import ShardRankGpu, run_lockstep
from tests.golden.make_golden import canon

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def test_norms_once_a_build(oracle_mod):
    import ctypes as C

    import torch

    n, R, L = 3_000, 24, 48
    first, second = D.gen_skewed_u8(n, 40, 30, 1), D.gen_skewed_u8(n, 40, 30, 2)
    gi = GpuIndex(np.uint8, "l2", n, 40, R)
    gi.upload_points(first)
    rank = ShardRankGpu(gi, L, 1.2)

    def launches_of_a_build():
        seen = []
        step = rank.search_prune

        def counted(lo, hi):
            rows = step(lo, hi)
            if hi > lo:
                seen.append(gi.launches())
            return rows

        rank.search_prune = counted
        run_lockstep([rank], rank.rounds)
        rank.search_prune = step
        return seen

    def check(points):
        og, _ = oracle_mod.build(points, R, L, 1.2)
        np.testing.assert_array_equal(canon(gi.graph()), canon(og))

    assert launches_of_a_build() == [3] + [2] * (len(rank.rounds) - 1)
    check(first)
    gi.upload_points(second)  # other points, same handle
    rank.begin()
    assert launches_of_a_build()[:2] == [3, 2]
    check(second)
    # points uploaded between dd_shard_begin and the first step
    rank.begin()
    rank.search_prune(0, 1)
    gi.upload_points(first)
    launches_of_a_build()
    check(first)
    # the caller holds the device points and may write them at any time
    base = C.c_void_p(gi.lib.dd_device_points(gi.h)).value
    stride = int(gi.lib.dd_device_row_stride(gi.h))

    class Rows:
        __cuda_array_interface__ = {"shape": (n, stride), "typestr": "|u1", "data": (base, False),
                                    "version": 3}

    rows = torch.as_tensor(Rows(), device="cuda")
    rank.begin()
    rank.search_prune(0, 1)
    rows[:, :40] = torch.from_numpy(second).cuda()
    torch.cuda.synchronize()
    launches_of_a_build()
    check(second)
    gi.close()
