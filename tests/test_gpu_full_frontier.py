"""Keyed searches whose frontier fills its whole array (beam widths 64, 128 and 256) in a
step of more than 32 candidates, the later of which lie beyond the frontier's last entry:
every entry of the final frontier, the visits and the counts are the oracle's and the plain
form's, for queries (k = L, few visits allowed) and for build searches."""
import numpy as np
import pytest

from distributed_diskann_b200 import datasets as D
from distributed_diskann_b200.index import GpuIndex

pytestmark = pytest.mark.gpu

NONE = 0xFFFFFFFF


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _chain(dtype, metric, L, R, kind, beyond, seed):
    """Points and a graph on which the search of point 1 visits point 0 (the start), then
    one hub after another; each hub's row is longer than the last hub's.  The last hub's
    row holds 32 entries of the final frontier and then `beyond` points that are farther
    than all L of it.  kind "fills": those 32 fill the frontier exactly; "trims": they
    fill it and push entries off; "full": it was full before them and the points beyond
    are still nearer than its old last entry.  The start is the frontier's last entry or
    (odd seeds) one in its middle."""
    rng = np.random.default_rng([seed, L, R, beyond])
    d = 24
    over = {"fills": 0, "trims": 7, "full": 0}[kind]
    good = L + over                       # ranks [0, good): the last row's 32 among them
    worse = 32 if kind == "full" else 0   # pushed off by them, beyond the points beyond
    need = good + beyond + worse
    pool = {"f32": rng.standard_normal((6 * need, d)).astype(np.float32),
            "i8": rng.integers(-128, 128, (6 * need, d)).astype(np.int8),
            "u8": rng.integers(0, 256, (6 * need, d)).astype(np.uint8)}[dtype]
    q = pool[-1]
    a, b = pool[:-1].astype(np.float64), q.astype(np.float64)
    dist = ((a - b) ** 2).sum(1) if metric == "l2" else -(a @ b)
    _, first = np.unique(dist, return_index=True)  # ascending, no two alike
    ranked = first[:need]
    far = ranked[good:good + beyond]
    start = ranked[good - 1] if seed % 2 == 0 else ranked[good // 2]
    entries = good + worse - 1 - 32       # what the rows before the last one hold
    nrows = -(-entries // min(R, 60))
    hubs = ranked[:nrows][::-1]           # every hub is nearer than all it was found with
    rest = [x for x in np.concatenate([ranked[nrows:good], ranked[good + beyond:]]) if x != start]
    rest = rng.permutation(rest)
    if kind == "full":                    # the worse ones come before the last row
        w = set(ranked[good + beyond:].tolist())
        rest = np.concatenate([[x for x in rest if x in w], [x for x in rest if x not in w]])
    rows, at = [], 0
    for i, part in enumerate(np.array_split(np.arange(entries - nrows), nrows)):
        rows.append(rng.permutation(np.concatenate([rest[at:at + len(part)], hubs[i:i + 1]])))
        at += len(part)
    rows.append(np.concatenate([rng.permutation(rest[at:]), rng.permutation(far)]))
    assert len(rest) - at == 32 and max(map(len, rows)) <= R
    ids = np.full(len(pool), NONE, np.uint32)   # pool row -> point id
    ids[start], ids[-1] = 0, 1
    others = [x for x in ranked if x != start]
    ids[others] = 2 + rng.permutation(len(others))
    n = 2 + len(others)
    base = np.zeros((n, d), pool.dtype)
    keep = ids != NONE
    base[ids[keep]] = pool[keep]
    graph = np.zeros((n, R + 1), np.uint32)
    for node, row in zip([start, *hubs], rows):
        graph[ids[node], 0] = len(row)
        graph[ids[node], 1:1 + len(row)] = ids[row]
    return base, graph, q[None], len(rows)


CHAINS = [("f32", "l2", 70), ("f32", "mips", 128), ("u8", "l2", 128), ("i8", "mips", 72)]


@pytest.mark.parametrize("kind", ["fills", "trims", "full"])
@pytest.mark.parametrize("L", [64, 128, 256])
@pytest.mark.parametrize("dtype,metric,R", CHAINS)
def test_query_candidates_beyond_a_full_frontier(oracle_mod, dtype, metric, R, L, kind):
    for seed, beyond in enumerate((1, 1, 2, 33, 38)):
        base, graph, q, visits = _chain(dtype, metric, L, R, kind, beyond, seed)
        gi = GpuIndex(base.dtype, metric, base.shape[0], base.shape[1], R)
        gi.upload_points(base)
        gi.set_graph(graph)
        for limit in (visits, 0):
            got = gi.search(q, L, L, limit=limit)
            gi.set_search_mode("plain")
            ref = gi.search(q, L, L, limit=limit)
            gi.set_search_mode("fast")
            for x, y in zip(got, ref):
                np.testing.assert_array_equal(x, y, err_msg=f"beyond={beyond} limit={limit}")
            oi, ov, oc = oracle_mod.search(base, graph, q, L, L, metric=metric, limit=limit)
            np.testing.assert_array_equal(got[0], oi)
            np.testing.assert_array_equal(got[2], ov)
            np.testing.assert_array_equal(got[3], oc)
        gi.close()


@pytest.mark.parametrize("kind", ["fills", "trims", "full"])
@pytest.mark.parametrize("L", [64, 128])
@pytest.mark.parametrize("dtype,metric", [("f32", "l2"), ("f32", "mips"), ("u8", "l2"),
                                          ("i8", "mips")])
def test_build_candidates_beyond_a_full_frontier(oracle_mod, dtype, metric, L, kind):
    """The build search of point 1 on the same graphs, through the sharded build's step:
    with an alpha that occludes nothing its new row is its visited list."""
    import torch

    from distributed_diskann_b200.sharded import ShardRankGpu

    R, alpha = 128, 500.0
    for seed, beyond in enumerate((1, 1, 2, 33, 38)):
        base, graph, _, _ = _chain(dtype, metric, L, R, kind, beyond, seed)
        want = oracle_mod.ShardRankOracle(base, R, L, alpha, metric=metric)
        want.graph[:] = graph
        row = want.search_prune(1, 2)[0]
        gi = GpuIndex(base.dtype, metric, base.shape[0], base.shape[1], R)
        gi.upload_points(base)
        for mode in ("plain", "fast"):
            rank = ShardRankGpu(gi, L, alpha, mode=mode)
            gi.set_graph(graph)
            got = rank.search_prune(1, 2)
            torch.cuda.synchronize()
            np.testing.assert_array_equal(got.cpu().numpy()[0, :row[0]].view(np.uint32),
                                          row[1:1 + row[0]], err_msg=f"{mode} beyond={beyond}")
        gi.close()


@pytest.mark.parametrize("dtype,metric,R,L", [
    ("f32", "l2", 40, 64), ("u8", "l2", 33, 64), ("i8", "mips", 64, 128), ("f32", "mips", 128, 128),
    ("i8", "l2", 100, 256), ("f32", "l2", 64, 256)])
def test_whole_frontiers_of_limited_searches(oracle_mod, dtype, metric, R, L):
    """Random rows, k = L, 2 to 10 visits: the frontier when the visits run out."""
    n, nq = 1_500, 150
    gen = {"f32": D.gen_mixture_f32, "i8": D.gen_mixture_i8, "u8": D.gen_skewed_u8}[dtype]
    both = gen(n + nq, 32, 12, R + L)
    base, q = both[:n], np.ascontiguousarray(both[n:])
    rng = np.random.default_rng(R)
    graph = np.zeros((n, R + 1), np.uint32)
    graph[:, 0] = rng.integers(33, R + 1, n)
    for i in range(n):
        graph[i, 1:1 + graph[i, 0]] = rng.choice(n, graph[i, 0], replace=False)
    gi = GpuIndex(base.dtype, metric, n, 32, R)
    gi.upload_points(base)
    gi.set_graph(graph)
    for limit in range(2, 11):
        ids, ds, vis, cm = gi.search(q, L, L, limit=limit)
        gi.set_search_mode("plain")
        ref = gi.search(q, L, L, limit=limit)
        gi.set_search_mode("fast")
        for x, y in zip((ids, ds, vis, cm), ref):
            np.testing.assert_array_equal(x, y, err_msg=f"limit={limit}")
        oi, ov, oc = oracle_mod.search(base, graph, q, L, L, metric=metric, limit=limit)
        found = np.isfinite(ds)
        np.testing.assert_array_equal(ids[found], oi[found])
        np.testing.assert_array_equal(vis, ov)
        np.testing.assert_array_equal(cm, oc)
    gi.close()


@pytest.mark.parametrize("dtype,R", [("f32", 64), ("u8", 128), ("i8", 40)])
@pytest.mark.parametrize("L", [64, 128])
def test_builds_of_few_points(oracle_mod, dtype, R, L):
    gen = {"f32": D.gen_mixture_f32, "i8": D.gen_mixture_i8, "u8": D.gen_skewed_u8}[dtype]
    for n in (100, 170, 256, 400):
        base = gen(n, 20, 5, n)
        og, ost = oracle_mod.build(base, R, L, 1.2)
        gi = GpuIndex(base.dtype, "l2", n, 20, R)
        gi.upload_points(base)
        st = gi.build(L, 1.2)
        g = gi.graph()
        for x in (g, og):
            x[:, 1:][np.arange(R)[None, :] >= x[:, :1]] = 0
        np.testing.assert_array_equal(g, og, err_msg=f"n={n}")
        assert st["visited"] == ost["visited"]
        gi.close()
