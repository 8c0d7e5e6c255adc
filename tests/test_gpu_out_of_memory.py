"""Calls that run out of device memory fail with an error and leave the handle usable, but
not before the idle buffers of earlier host calls are given back."""
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


def test_idle_buffers_of_host_calls_are_given_back():
    """A float ground truth leaves a buffer of 300 MB; calls of the same handle and of
    others then find less free memory than they need."""
    import torch

    n, d = 300_000, 256
    base = torch.randn(n, d, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    q = base[:40].cpu().numpy()
    gi = GpuIndex(np.float32, "l2", n, d, 64)
    gi.upload_points(base)
    torch.cuda.synchronize()
    del base
    small = D.gen_mixture_f32(200_000, 64, 60, 3)

    def ground_truth():
        ids, _ = gi.groundtruth(q, 3)
        np.testing.assert_array_equal(ids[:, 0], np.arange(40))

    ground_truth()
    with free_memory(40):
        g = gi.graph()  # 78 MB of rows
    assert not g.any()
    ground_truth()
    with free_memory(40):
        other = GpuIndex(small.dtype, "l2", 200_000, 64, 64)  # 102 MB
        other.upload_points(small)
    ground_truth()
    with free_memory(60):
        other.build(64, 1.2, max_build=20_000)  # 100 MB of scratch
        ids = other.search(small[:50], 1, 20, skip_self=False)[0]
    want = GpuIndex(small.dtype, "l2", 200_000, 64, 64)
    want.upload_points(small)
    want.build(64, 1.2, max_build=20_000)
    np.testing.assert_array_equal(ids, want.search(small[:50], 1, 20, skip_self=False)[0])
    for x in (gi, other, want):
        x.close()


@pytest.mark.parametrize("work_mb", [400, 40, 8, 0])
@pytest.mark.parametrize("kind", ["u8", "i8", "f32", "ties", "mips"])
def test_ground_truth_of_a_bounded_workspace(oracle_mod, monkeypatch, kind, work_mb):
    """Batches of queries (float ones with queries left to the FP64 form on both sides of
    each boundary), slabs of 8192 rows and up, one CTA and more."""
    rng = np.random.default_rng(5)
    n, nq, d = 20_001, 1_300, 24
    metric = "mips" if kind == "mips" else "l2"
    if kind in ("u8", "i8"):
        t, lo = (np.uint8, 0) if kind == "u8" else (np.int8, -128)
        base = rng.integers(lo, lo + 256, (n, d)).astype(t)
        q = rng.integers(lo, lo + 256, (nq, d)).astype(t)
    else:
        base = rng.standard_normal((n, d), dtype=np.float32)
        q = rng.standard_normal((nq, d), dtype=np.float32)
        if kind == "ties":  # hundreds of points at one distance of every third query
            base = rng.integers(0, 3, (n, d)).astype(np.float32)
            q[::3] = rng.integers(0, 3, (len(q[::3]), d))
    monkeypatch.setenv("DD_GT_WORK_BYTES", str(work_mb * MB))
    gi = GpuIndex(base.dtype, metric, n, d, 8)
    gi.upload_points(base)
    for k in (32, 3):
        ids, ds = gi.groundtruth(q, k)
        oi, od = oracle_mod.groundtruth(base, q, k, metric=metric)
        np.testing.assert_array_equal(ids, oi)
        np.testing.assert_array_equal(ds, od)
    gi.close()


@pytest.mark.parametrize("dtype,nq", [("f32", 300), ("u8", 3_000)])
def test_ground_truth_with_little_memory_left(dtype, nq):
    """A workspace of 310 MB (float rows as BF16 halves) or 60 MB (candidate lists) does
    not fit; a smaller one gives the same answer."""
    import torch

    n, d = 300_000, 256
    g = torch.Generator("cuda").manual_seed(2)
    if dtype == "f32":
        base = torch.randn(n, d, device="cuda", generator=g)
    else:
        base = torch.randint(0, 256, (n, d), device="cuda", generator=g, dtype=torch.uint8)
    q = base[:nq].cpu().numpy()
    gi = GpuIndex(np.dtype(np.float32 if dtype == "f32" else np.uint8), "l2", n, d, 8)
    gi.upload_points(base)
    torch.cuda.synchronize()
    del base
    with free_memory(100 if dtype == "f32" else 24):
        ids, ds = gi.groundtruth(q, 10)
    wi, wd = gi.groundtruth(q, 10)
    np.testing.assert_array_equal(ids, wi)
    np.testing.assert_array_equal(ds, wd)
    gi.close()


def _mixed_search():
    both = D.gen_mixture_f32(35_000, 24, 40, 3)
    base, q = both[:5_000], both[5_000:]
    Ls = np.resize(np.array([10, 20, 50, 100, 200], np.uint32), len(q))

    def handle():
        gi = GpuIndex(base.dtype, "l2", 5_000, 24, 24)
        gi.upload_points(base)
        gi.build(48, 1.2)
        return gi

    return handle, q, Ls


def test_a_search_whose_scratch_does_not_fit_fails():
    handle, q, Ls = _mixed_search()
    gi = handle()
    with free_memory(40):
        for _ in range(2):
            with pytest.raises(DDError, match="memory"):
                gi.search(q, 10, Ls)
    got = gi.search(q, 10, Ls)
    gi.close()
    gi = handle()
    for a, b in zip(gi.search(q, 10, Ls), got):
        np.testing.assert_array_equal(a, b)
    gi.close()


def test_mixed_widths_with_little_memory_left():
    """Scratch for classes that overlap does not fit; the classes run one by one."""
    import torch

    handle, q, Ls = _mixed_search()
    gi = handle()
    torch.cuda.empty_cache()
    before, _ = torch.cuda.mem_get_info()
    want = gi.search(q, 10, Ls)
    need = (before - torch.cuda.mem_get_info()[0]) // MB
    gi.close()
    gi = handle()
    gi.search(q[:5], 10, 200)  # (a first call of few queries)
    with free_memory(need * 3 // 4):
        got = gi.search(q, 10, Ls)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(gi.search(q, 10, Ls), want):
        np.testing.assert_array_equal(a, b)
    gi.close()
