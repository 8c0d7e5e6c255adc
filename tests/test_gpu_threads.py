"""Handles of several shapes called from several threads at once: kernels that they share
are launched with different amounts of shared memory in between."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from distributed_diskann_b200 import datasets as D
from distributed_diskann_b200.index import GpuIndex

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def test_calls_of_several_shapes_from_several_threads():
    def answers(d):
        both = D.gen_mixture_i8(1_540, d, 20, d)
        base, q = both[:1_500], np.ascontiguousarray(both[1_500:])
        out = []
        gi = GpuIndex(base.dtype, "l2", 1_500, d, 16)
        gi.upload_points(base)
        gi.build(32, 1.2)
        for r in range(60):
            L = (20, 100, 200, 300)[(r + d) % 4]
            out += [gi.groundtruth(q, 3)[0], gi.search(q, 5, L)[0],
                    gi.robust_prune([(1, np.arange(50 + d, dtype=np.uint32),
                                      np.arange(50 + d, dtype=np.float32))], 1.2)[0]]
        gi.close()
        return out

    dims = (10, 70, 130, 200, 300, 500, 700, 1000)
    want = [answers(d) for d in dims]
    for _ in range(3):
        with ThreadPoolExecutor(len(dims)) as pool:
            for w, g in zip(want, pool.map(answers, dims)):
                assert len(w) == len(g)
                for a, b in zip(w, g):
                    np.testing.assert_array_equal(a, b)
