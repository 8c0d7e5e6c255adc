"""The fast query search at the edges of its frontier sizes (64, 128, 256 entries, the
id/distance form beyond), with visit and degree limits, every k-cut, both metrics, and
on graphs whose rows repeat ids (the search then has to fall back: frontiers become
multisets, and a repeated candidate may already be in the frontier or be pushed off at
once).  Ids, visits and distance counts are the oracle's, and the plain form's."""
import numpy as np
import pytest

from distributed_diskann_b200 import datasets as D
from distributed_diskann_b200.index import GpuIndex

pytestmark = pytest.mark.gpu

WIDTHS = (10, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 400)


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("repeats", [False, True])
@pytest.mark.parametrize("dtype,metric,d,R", [("u8", "l2", 32, 24), ("i8", "mips", 48, 70),
                                              ("f32", "l2", 20, 40), ("f32", "mips", 37, 24)])
def test_query_widths_and_repeated_ids(oracle_mod, dtype, metric, d, R, repeats):
    n, nq = 3_000, 60
    gen = {"f32": D.gen_mixture_f32, "i8": D.gen_mixture_i8, "u8": D.gen_skewed_u8}[dtype]
    both = gen(n + nq, d, 12, 9 + d)
    both[n // 2:n // 2 + 200] = both[:200]  # equal distances, and zero ones for the k-cut
    base, q = both[:n], both[n:].copy()
    q[:5] = base[7:12]
    rng = np.random.default_rng(R)
    graph = np.zeros((n, R + 1), np.uint32)
    graph[:, 0] = rng.integers(1, R + 1, n)
    graph[:, 1:] = rng.integers(0, n, (n, R))  # chance repeats
    for i in range(n):
        deg = graph[i, 0]
        row = rng.choice(n, deg, replace=False)
        if repeats and i % 3 == 0 and deg > 4:
            row[deg // 2:] = row[: deg - deg // 2][rng.permutation(deg - deg // 2)]
        graph[i, 1:1 + deg] = row
        graph[i, 1 + deg:] = 0
    gi = GpuIndex(base.dtype, metric, n, d, R)
    gi.upload_points(base)
    gi.set_graph(graph)
    for L in WIDTHS:
        for k, cut, limit, dlim in ((10, 1.35, 0, 0), (3, 1.0, 0, R // 2), (1, 1.35, 7, 0)):
            got = gi.search(q, k, L, cut=cut, limit=limit, degree_limit=dlim)
            gi.set_search_mode("plain")
            ref = gi.search(q, k, L, cut=cut, limit=limit, degree_limit=dlim)
            gi.set_search_mode("fast")
            for a, b in zip(got, ref):
                np.testing.assert_array_equal(a, b, err_msg=f"L={L} k={k} cut={cut} limit={limit}")
        if L in (33, 128, 129):
            oi, ov, oc = oracle_mod.search(base, graph, q, 10, L, metric=metric)
            ids, ds, vis, cm = gi.search(q, 10, L)
            np.testing.assert_array_equal(vis, ov)
            np.testing.assert_array_equal(cm, oc)
            found = np.isfinite(ds)
            np.testing.assert_array_equal(ids[found], oi[found])
    gi.close()


@pytest.mark.parametrize("dtype", ["u8", "f32"])
@pytest.mark.parametrize("nq,widths", [
    (3, (10, 200)), (900, (10, 20, 50, 100, 200)),       # one launch of the widest layout
    (9_000, (10, 20, 50, 100, 200)),                     # overlapped classes, two groups
    (4_000, (500, 10, 300, 130, 70, 40, 20, 12)),        # every class
])
def test_mixed_widths_in_one_call(dtype, nq, widths):
    """One call of several beam widths, from the host and on the device (where the
    widths are unknown to the launch), against a call of each width alone."""
    import torch

    gen = {"f32": D.gen_mixture_f32, "u8": D.gen_skewed_u8}[dtype]
    both = gen(4_000 + nq, 32, 15, 4)
    base, q = both[:4_000], np.ascontiguousarray(both[4_000:])
    gi = GpuIndex(base.dtype, "l2", 4_000, 32, 32)
    gi.upload_points(base)
    gi.build(64, 1.2)
    Ls = np.resize(np.asarray(widths, np.uint32), nq)
    want = [None, np.zeros((nq, 10), np.float32), np.zeros(nq, np.uint32), np.zeros(nq, np.uint32)]
    want[0] = np.zeros((nq, 10), np.uint32)
    for w in widths:
        for a, b in zip(want, gi.search(q, 10, int(w))):
            a[Ls == w] = b[Ls == w]
    for _ in range(2):
        for a, b in zip(want, gi.search(q, 10, Ls)):
            np.testing.assert_array_equal(a, b)
    dq = torch.from_numpy(q).cuda()
    dL = torch.from_numpy(Ls.view(np.int32)).cuda()
    out = [torch.zeros((nq, 10), dtype=torch.int32, device="cuda"),
           torch.zeros((nq, 10), device="cuda"),
           torch.zeros(nq, dtype=torch.int32, device="cuda"),
           torch.zeros(nq, dtype=torch.int32, device="cuda")]
    torch.cuda.synchronize()
    gi.search_device(dq.data_ptr(), nq, dq.stride(0) * dq.element_size(), dL.data_ptr(),
                     max(widths), 10, out[0].data_ptr(), out[1].data_ptr(),
                     vis_ptr=out[2].data_ptr(), cmps_ptr=out[3].data_ptr())
    torch.cuda.synchronize()
    for a, b in zip(want, out):
        np.testing.assert_array_equal(a.view(np.int32), b.cpu().numpy().view(np.int32))
    gi.close()
