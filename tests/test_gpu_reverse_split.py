"""Reverse edges of the fast form's large rounds: targets split into appends, short
prunes (only pairs with a new entry), general prunes and hub targets.  Graphs must be
the oracle's, bit for bit, at row widths on both sides of every form's limit: one and
two 64-byte halves, odd widths, integer rows beyond the tensor-core form (129), float
rows in registers (64) and beyond (65), degrees up to the row capacity (lists beyond
128 candidates), and a second pass with another alpha (no row counts as pruned)."""
import numpy as np
import pytest

from distributed_diskann_b200 import datasets as D
from distributed_diskann_b200.index import GpuIndex
from tests.golden.make_golden import canon

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _points(dtype, metric, n, d, seed):
    if dtype == "f32":
        x = D.gen_mixture_f32(n, d, 6, seed)
        if metric == "mips":
            x /= np.linalg.norm(x, axis=1, keepdims=True)
        return np.ascontiguousarray(x, np.float32)
    return (D.gen_mixture_i8 if dtype == "i8" else D.gen_skewed_u8)(n, d, 6, seed)


@pytest.mark.parametrize("dtype,metric,d,R,xita,two_pass", [
    ("u8", "l2", 1, 32, 1.0, False), ("u8", "l2", 64, 64, 0.3, False),
    ("u8", "l2", 65, 32, 1.0, False), ("u8", "l2", 128, 64, 0.3, False),
    ("u8", "l2", 129, 32, 1.0, False), ("u8", "mips", 33, 32, 1.0, False),
    ("i8", "l2", 100, 128, 0.3, False), ("i8", "l2", 100, 64, 0.15, False),
    ("i8", "l2", 30, 30, 1.0, True), ("i8", "mips", 100, 32, 1.0, False),
    ("f32", "l2", 64, 48, 0.3, False), ("f32", "l2", 65, 32, 1.0, False),
    ("f32", "l2", 3, 32, 1.0, True), ("f32", "mips", 40, 32, 0.5, False),
])
def test_split_rounds_give_the_oracle_graph(oracle_mod, dtype, metric, d, R, xita, two_pass):
    n = 5_000
    base = _points(dtype, metric, n, d, 100 + d + R)
    kw = {"knn_mode": True, "two_pass": True} if two_pass else {}
    gi = GpuIndex(base.dtype, metric, n, d, R)
    gi.upload_points(base)
    st = gi.build(2 * R if R < 100 else 128, 1.2, max_fraction=xita, **kw)
    graph = canon(gi.graph())
    okw = {"knn_mode": True, "two_pass": True} if two_pass else {"xita": xita}
    og, ost = oracle_mod.build(base, R, 2 * R if R < 100 else 128, 1.2, metric=metric, **okw)
    np.testing.assert_array_equal(graph, canon(og))
    for k in ("groups", "reverse_prunes", "prune_cands"):
        assert st[k] == ost[k]
    assert st["reverse_prunes"] > 0
    gi.close()
