"""Ground truth on the tensor cores against the oracle at the edges of its tiles: one
query and one more than a query tile, base sizes around a tile of 128 points, rows of
one and of several k-blocks, odd widths, k of 1 and 32, several slabs of float rows, and
float queries the BF16 screen must hand to the FP64 form (ties beyond a list's capacity,
values whose bound overflows, subnormal values).  Distances and ids are exact: float
candidates get the FP64 distance of the definition, integers are exact."""
import numpy as np
import pytest

from distributed_diskann_b200.index import GpuIndex

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _check(oracle_mod, base, q, metric, ks):
    gi = GpuIndex(base.dtype, metric, base.shape[0], base.shape[1], 8)
    gi.upload_points(base)
    for k in ks:
        ids, ds = gi.groundtruth(q, k)
        oi, od = oracle_mod.groundtruth(base, q, k, metric=metric)
        np.testing.assert_array_equal(ids, oi)
        np.testing.assert_array_equal(ds, od)
    gi.close()


@pytest.mark.parametrize("metric", ["l2", "mips"])
@pytest.mark.parametrize("dtype,n,nq,d", [
    ("u8", 32, 1, 1), ("u8", 127, 256, 128), ("u8", 129, 257, 129), ("u8", 40_001, 3, 128),
    ("i8", 128, 129, 64), ("i8", 9_000, 300, 65), ("i8", 3_000, 7, 1024), ("u8", 3_000, 130, 1000),
    ("f32", 32, 1, 1), ("f32", 127, 128, 16), ("f32", 129, 129, 17), ("f32", 20_000, 131, 200),
    ("f32", 5_000, 9, 256), ("f32", 30_011, 500, 64),
])
def test_tile_edges(oracle_mod, metric, dtype, n, nq, d):
    rng = np.random.default_rng(n + nq + d)
    if dtype == "f32":
        base = rng.standard_normal((n, d), dtype=np.float32)
        q = rng.standard_normal((nq, d), dtype=np.float32)
    else:
        lo, hi = (-128, 128) if dtype == "i8" else (0, 256)
        t = np.int8 if dtype == "i8" else np.uint8
        base = rng.integers(lo, hi, (n, d)).astype(t)
        q = rng.integers(lo, hi, (nq, d)).astype(t)
        base[: n // 4] = hi - 1 if dtype == "u8" else lo  # the largest norms and products
    _check(oracle_mod, base, q, metric, (32, 1))


@pytest.mark.parametrize("metric", ["l2", "mips"])
@pytest.mark.parametrize("kind", ["ties", "huge", "tiny", "outlier", "clusters"])
def test_float_queries_the_screen_cannot_bound(oracle_mod, metric, kind):
    rng = np.random.default_rng(3)
    n, nq, d = 6_000, 70, 24
    base = rng.standard_normal((n, d), dtype=np.float32)
    q = rng.standard_normal((nq, d), dtype=np.float32)
    if kind == "ties":  # values 0..2: hundreds of points at one distance
        base = rng.integers(0, 3, (n, d)).astype(np.float32)
        q[:35] = rng.integers(0, 3, (35, d))
    elif kind == "huge":
        base *= np.float32(3e17)
        q *= np.float32(3e17)
    elif kind == "tiny":
        base *= np.float32(1e-22)
        q *= np.float32(1e-22)
    elif kind == "outlier":  # one base row's norm widens every bound
        base[17] *= np.float32(3e6)
    else:  # tight clusters around far centres
        cent = (rng.standard_normal((20, d)) * 50).astype(np.float32)
        base = cent[rng.integers(0, 20, n)] + base * np.float32(0.01)
        q = cent[rng.integers(0, 20, nq)] + q * np.float32(0.01)
    _check(oracle_mod, np.ascontiguousarray(base), np.ascontiguousarray(q), metric, (10, 32))


def test_several_slabs_of_float_rows(oracle_mod):
    rng = np.random.default_rng(11)
    base = rng.standard_normal((1_100_000, 5), dtype=np.float32)
    q = rng.standard_normal((20, 5), dtype=np.float32)
    base[1_050_000:1_050_020] = q  # the nearest ones lie in the second slab
    _check(oracle_mod, base, q, "l2", (10,))


@pytest.mark.parametrize("metric", ["l2", "mips"])
@pytest.mark.parametrize("dtype,d", [("u8", 64), ("i8", 200), ("f32", 24)])
def test_lists_that_fill_up(oracle_mod, metric, dtype, d):
    """31 tiles (no sample), several a CTA, the rows ever nearer: every value passes its
    query's threshold until the list is compacted."""
    rng = np.random.default_rng(d)
    n, nq = 31 * 128 - 5, 2_600
    t = {"u8": np.uint8, "i8": np.int8, "f32": np.float32}[dtype]
    base = np.zeros((n, d), t)
    base += (np.arange(n) * (100.0 / n)).astype(t)[:, None]
    base[:, 0] = rng.integers(0, 100, n)
    q = (100 + rng.integers(0, 20, (nq, d))).astype(t)
    _check(oracle_mod, base, q, metric, (32, 5))


def test_more_queries_than_one_workspace():
    rng = np.random.default_rng(12)
    n, nq, d, k = 4_000, 1_500_001, 4, 3
    base = rng.integers(0, 256, (n, d)).astype(np.uint8)
    q = rng.integers(0, 256, (nq, d)).astype(np.uint8)
    gi = GpuIndex(base.dtype, "l2", n, d, 8)
    gi.upload_points(base)
    ids, ds = gi.groundtruth(q, k)
    for pick in (slice(0, 1000), slice(nq // 2 - 500, nq // 2 + 500),
                 slice(nq // 4 - 500, nq // 4 + 500), slice(nq - 1000, nq)):
        wi, wd = gi.groundtruth(q[pick], k)
        np.testing.assert_array_equal(ids[pick], wi)
        np.testing.assert_array_equal(ds[pick], wd)
    gi.close()
