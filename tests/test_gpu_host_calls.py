"""Host calls keep one device buffer per handle and share pinned staging, and search only the
beam-width classes a call holds: calls of growing and shrinking sizes, strided query
rows, one and several classes, calls that fail in between, and prunes on both sides of
the shared-memory limit must give what the oracle (or a fresh handle) gives."""
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


@pytest.mark.parametrize("dtype", ["i8", "f32"])
def test_calls_of_changing_size_on_one_handle(oracle_mod, dtype):
    gen = D.gen_mixture_i8 if dtype == "i8" else D.gen_mixture_f32
    both = gen(5_000, 30, 20, 5)  # 30 bytes / 120 bytes a row: padded on the device
    base, q = both[:4_000], both[4_000:]
    gi = GpuIndex(base.dtype, "l2", 4_000, 30, 24)
    gi.upload_points(base)
    gi.build(48, 1.2)
    g = gi.graph()
    for nq, L in ((1, 20), (700, [10, 20, 50, 100, 200, 64, 17]), (3, [10, 300, 12]), (1000, 100),
                  (2, 16)):
        Ls = np.broadcast_to(np.asarray(L, np.uint32), (nq,)) if np.isscalar(L) else np.resize(
            np.asarray(L, np.uint32), nq)
        ids, _, vis, cm = gi.search(q[:nq], 10, Ls)
        for w in sorted(set(Ls.tolist())):
            oi, ov, oc = oracle_mod.search(base, g, q[:nq], 10, int(w))
            s = Ls == w
            np.testing.assert_array_equal(ids[s], oi[s])
            np.testing.assert_array_equal(vis[s], ov[s])
            np.testing.assert_array_equal(cm[s], oc[s])
        with pytest.raises(DDError):
            gi.search(q[:nq], 10, 5)  # k above the beam width
        ti, td = gi.groundtruth(q[:nq], 5)
        oi, od = oracle_mod.groundtruth(base, q[:nq], 5)
        np.testing.assert_array_equal(ti, oi)
        np.testing.assert_array_equal(td, od)
    # rows further apart than their length
    wide = np.zeros((50, 64), base.dtype)
    wide[:, :30] = q[:50]
    Ls = np.full(50, 40, np.uint32)
    ids, ds = np.zeros((50, 10), np.uint32), np.zeros((50, 10), np.float32)
    p = lambda a: C.c_void_p(a.ctypes.data)
    gi._ck(gi.lib.dd_search(gi.h, p(wide), 50, wide.strides[0], p(Ls), 10, 1.35, 0, 0, 0, 1, p(ids),
                            p(ds), None, None))
    np.testing.assert_array_equal(ids, gi.search(q[:50], 10, 40)[0])
    gi.close()


def test_handles_of_several_threads_share_the_staging():
    """Handles opened, called and closed by threads at once, calls of growing and
    shrinking size: the answers of one handle used alone."""
    from concurrent.futures import ThreadPoolExecutor

    both = D.gen_mixture_i8(6_000, 24, 20, 6)
    base, q = both[:3_000], both[3_000:]
    sizes = (1, 2_900, 40, 900, 3)

    def answers(seed):
        out = []
        for again in range(2):
            gi = GpuIndex(base.dtype, "l2", 3_000, 24, 16)
            gi.upload_points(base)
            gi.build(32, 1.2)
            for nq in sizes[seed:] + sizes[:seed]:
                r = gi.search(q[:nq], 5, 20)
                out.append((nq, r[0].copy(), gi.groundtruth(q[:nq], 3)[0]))
            gi.close()
        return sorted(out, key=lambda r: r[0])

    want = answers(0)
    with ThreadPoolExecutor(4) as pool:
        for got in pool.map(answers, range(4)):
            for w, g in zip(want, got):
                np.testing.assert_array_equal(w[1], g[1])
                np.testing.assert_array_equal(w[2], g[2])


@pytest.mark.parametrize("dtype,metric,d", [("u8", "l2", 128), ("i8", "mips", 20),
                                            ("u8", "l2", 200), ("f32", "l2", 64),
                                            ("f32", "mips", 90)])
@pytest.mark.parametrize("most", [1, 40, 700, 6_000])
def test_prunes_in_shared_and_in_global_memory(oracle_mod, dtype, metric, d, most):
    """Keys the caller made up (infinite ones, ties, fractions among them), rows of the
    graph taken in, alpha of 0.5 to 2: the oracle's lists."""
    rng = np.random.default_rng(d + most)
    n, R = 8_000, 20
    if dtype == "f32":
        base = rng.standard_normal((n, d), dtype=np.float32)
    else:
        base = (rng.integers(0, 256, (n, d)).astype(np.uint8) if dtype == "u8"
                else rng.integers(-128, 128, (n, d)).astype(np.int8))
    gi = GpuIndex(base.dtype, metric, n, d, R)
    gi.upload_points(base)
    graph = np.zeros((n, R + 1), np.uint32)
    graph[:, 0] = rng.integers(0, R + 1, n)
    graph[:, 1:] = rng.integers(0, n, (n, R))
    graph[:, 1:][np.arange(R)[None, :] >= graph[:, :1]] = 0
    gi.set_graph(graph)
    for alpha in (1.2, 0.5, 2.0):
        tasks = []
        for t in range(25):
            m = int(rng.integers(0, most + 1)) if t else most
            keys = (rng.standard_normal(m) * 1e4).astype(np.float32)
            keys[rng.random(m) < 0.2] = np.float32(77.25)
            keys[rng.random(m) < 0.02] = np.float32(np.inf)
            tasks.append((int(rng.integers(n)), rng.integers(0, n, m).astype(np.uint32), keys))
        outs = gi.robust_prune(tasks, alpha)
        for t, (p, ids, keys) in enumerate(tasks):
            exp = oracle_mod.robust_prune(base, graph, p, ids, keys, alpha, metric=metric)
            np.testing.assert_array_equal(outs[t], exp, err_msg=f"task {t}")
    gi.close()
