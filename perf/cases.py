"""The work this framework is measured on: index builds, query searches, ground truth
and prunes, through its public entry points.

Sizes are those of the repository's own workloads (10,000 x 20 f32, 100,000 x 64 f32,
1M x 100 int8, 1M x 200 f32 inner product, N x 128 uint8) or generic ones; points come
from the same distributions as ``distributed_diskann_b200.datasets``, drawn on the GPU.

A case is a dict of plain values.  ``kind`` says which entry point it goes through:

  bsp     BSPIndex.bsp_build: host points in, host graph out, a fresh index each time
  build   GpuIndex.build on resident points; the graph is read through the device view
  search  GpuIndex.search: host queries, host results
  dsearch GpuIndex.search_device: device queries, device results
  gt      GpuIndex.groundtruth: host queries, host results
  prune   GpuIndex.robust_prune: candidate lists in, selected ids out
"""
import numpy as np
import torch

from distributed_diskann_b200.index import (BSPIndex, BuildParams, DatasetPara, Graph, GpuIndex,
                                            PointRange)

DEV = "cuda"
NP = {"f32": np.float32, "i8": np.int8, "u8": np.uint8}
ESZ = {"f32": 4, "i8": 1, "u8": 1}


def _build(name, kind, dtype, metric, n, d, R, L, alpha, xita, knn=False, two_pass=False):
    return {"name": name, "kind": kind, "dtype": dtype, "metric": metric, "n": n, "d": d, "R": R,
            "L": L, "alpha": alpha, "xita": xita, "knn": knn, "two_pass": two_pass}


def _search(name, kind, dtype, metric, n, d, R, Lb, alpha, nq, k, beam, limit=0, degree_limit=0):
    return {"name": name, "kind": kind, "dtype": dtype, "metric": metric, "n": n, "d": d, "R": R,
            "L": Lb, "alpha": alpha, "nq": nq, "k": k, "beam": beam, "limit": limit,
            "degree_limit": degree_limit}


def _gt(name, dtype, metric, n, d, nq, k):
    return {"name": name, "kind": "gt", "dtype": dtype, "metric": metric, "n": n, "d": d,
            "nq": nq, "k": k}


def _prune(name, dtype, metric, n, d, R, Lb, alpha, tasks):
    return {"name": name, "kind": "prune", "dtype": dtype, "metric": metric, "n": n, "d": d,
            "R": R, "L": Lb, "alpha": alpha, "tasks": tasks}


def listed():
    return [
        # one query of an interactive caller: the latency of a call
        _search("search-one", "search", "f32", "l2", 100_000, 64, 48, 96, 1.2, 1, 10, 100),
        # the query sweep of the uint8 workload at its recall width, device to device
        _search("search-u8", "dsearch", "u8", "l2", 1_000_000, 128, 64, 128, 1.2, 10_000, 10, 100),
        # a batch of requests of every beam width of the sweep (beam 0: 10, 20, 50, 100, 200)
        _search("search-i8-mixed", "search", "i8", "l2", 1_000_000, 100, 64, 128, 1.2, 30_000, 10,
                0),
        # inner-product search of long float rows, a large batch
        _search("search-mips", "dsearch", "f32", "mips", 400_000, 200, 64, 128, 1.0, 50_000, 10,
                50),
        # the drop-in build of the shipped small set: host to host, fresh index, 2% rounds
        _build("bsp-xs", "bsp", "f32", "l2", 10_000, 20, 32, 64, 1.2, 0.02),
        # a mid-size float build in doubling rounds
        _build("build-f32", "build", "f32", "l2", 100_000, 64, 48, 96, 1.2, 1.0),
        # the int8 workload with the parameter file's default 2% rounds (many small rounds)
        _build("build-i8", "build", "i8", "l2", 1_000_000, 100, 64, 128, 1.2, 0.02),
        # the inner-product workload's build: long float rows, alpha 1
        _build("build-mips", "build", "f32", "mips", 400_000, 200, 64, 128, 1.0, 1.0),
        # the largest: the uint8 workload at 4M points, rounds up to a million
        _build("build-u8", "build", "u8", "l2", 4_000_000, 128, 64, 128, 1.2, 1.0),
        # exact neighbours for the recall of the uint8 queries
        _gt("gt-u8", "u8", "l2", 1_000_000, 128, 10_000, 32),
        # exact neighbours of float inner-product queries
        _gt("gt-mips", "f32", "mips", 400_000, 200, 1_000, 32),
        # robustPrune called on its own: the visited lists of a few hundred points
        _prune("prune-i8", "i8", "l2", 100_000, 100, 64, 128, 1.2, 512),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _unnamed(case):
    return {k: v for k, v in case.items() if k != "name"}


def draw(rng):
    """One more case: any kind, sizes spread over the ranges of the listed ones."""
    kind = rng.choice(["build", "build", "bsp", "search", "search", "dsearch", "gt", "gt", "prune"])
    dtype = rng.choice(["f32", "i8", "u8"])
    metric = rng.choice(["l2", "l2", "mips"]) if dtype == "f32" else "l2"
    d = _log(rng, 10, 200) if dtype == "f32" else _log(rng, 20, 200)
    R = rng.choice([24, 32, 48, 50, 64])
    L = R * 2
    alpha = 1.0 if metric == "mips" else 1.2
    if kind == "gt":
        nq = _log(rng, 10, 10_000)
        most = 4e11 if dtype == "f32" else 2e12
        n = max(1_000, min(_log(rng, 5_000, 1_000_000), int(most / 2 / nq / d)))
        return _unnamed(_gt("", dtype, metric, n, d, nq, rng.choice([10, 32])))
    if kind == "build":
        n = _log(rng, 3_000, 300_000 if dtype == "f32" else 1_000_000)
        knn = rng.random() < 0.25
        two_pass = knn and n < 200_000 and rng.random() < 0.5
        return _unnamed(_build("", "build", dtype, metric, n, d, R, L, alpha,
                               1.0 if knn else rng.choice([0.02, 1.0]), knn, two_pass))
    if kind == "bsp":
        return _unnamed(_build("", "bsp", dtype, metric, _log(rng, 1_000, 100_000), d, R, L, alpha,
                               rng.choice([0.02, 1.0])))
    n = _log(rng, 5_000, 400_000)
    if kind == "prune":
        return _unnamed(_prune("", dtype, metric, n, d, R, L, alpha, _log(rng, 1, 2_000)))
    nq = _log(rng, 1, 30_000)
    beam = rng.choice([0, 10, 20, 50, 100, 200, _log(rng, 12, 300)])
    limit = rng.choice([0, 0, 0, 64])
    return _unnamed(_search("", kind, dtype, metric, n, d, R, L, alpha, nq, 10, beam, limit,
                            rng.choice([0, 0, 0, R // 2])))


# ------------------------------------------------------------------ inputs
def _points(case, total, seed):
    """`total` rows of the case's distribution on the GPU (a Gaussian mixture)."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    d, dtype = case["d"], case["dtype"]
    ncent = max(10, min(10_000, case["n"] // 500))
    rows = torch.empty((total, d), device=DEV, dtype=getattr(torch, {"f32": "float32", "i8": "int8",
                                                                     "u8": "uint8"}[dtype]))
    cent = torch.randn((ncent, d), device=DEV, generator=g)
    if dtype != "f32":
        cent *= 40.0
        if dtype == "u8":
            cent = cent.abs()
    elif case["metric"] == "l2":
        cent = torch.rand((ncent, d), device=DEV, generator=g) * 20.0 - 10.0
    step = 1 << 19
    for s in range(0, total, step):
        m = min(step, total - s)
        v = cent[torch.randint(0, ncent, (m,), device=DEV, generator=g)]
        noise = torch.randn((m, d), device=DEV, generator=g)
        if dtype == "u8":
            v = (v + 12.0 * noise).abs().round().clamp(0, 255)
        elif dtype == "i8":
            v = (v + 12.0 * noise).round().clamp(-128, 127)
        elif case["metric"] == "l2":
            v = v + noise
        else:
            v = torch.nn.functional.normalize(v + 0.3 * noise, dim=1)
        rows[s:s + m] = v.to(rows.dtype)
    return rows


def _sets(case, seed):
    """Base and query rows on the GPU."""
    nq = case.get("nq", 0)
    both = _points(case, case["n"] + nq, seed)
    q = both[case["n"]:]
    if nq and case["metric"] == "mips":
        g = torch.Generator(device=DEV)
        g.manual_seed(seed + 1)
        q = torch.nn.functional.normalize(
            q + 0.3 * torch.randn(q.shape, device=DEV, generator=g) / case["d"] ** 0.5, dim=1)
    return both[:case["n"]], q


def _index(case, base, R):
    gi = GpuIndex(NP[case["dtype"]], case["metric"], case["n"], case["d"], R)
    gi.upload_points(base)
    torch.cuda.synchronize()
    return gi


class _DeviceRows:
    """The index's graph rows on the device, for torch.as_tensor."""

    def __init__(self, gi):
        self.gi = gi  # the rows live as long as the index
        self.__cuda_array_interface__ = {
            "shape": (gi.n, int(gi.lib.dd_device_row_len(gi.h))), "typestr": "<i4",
            "data": (int(gi.lib.dd_device_graph(gi.h)), False), "version": 3}


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    base, q = _sets(case, seed)
    if kind == "bsp":
        s["points"] = PointRange(base.cpu().numpy(), metric=case["metric"])
        s["bp"] = BuildParams(case["R"], case["L"], case["alpha"])
        dp = DatasetPara()
        dp.alpha, dp.xita, dp.save = case["alpha"], case["xita"], False
        s["dp"] = dp
        return s
    gi = s["gi"] = _index(case, base, case.get("R", 32))
    if kind == "build":
        s["graph"] = torch.as_tensor(_DeviceRows(gi), device=DEV)
        return s
    if kind == "gt":
        s["queries"] = q.cpu().numpy()
        return s
    gi.build(case["L"], case["alpha"], collect_stats=False)
    if kind == "prune":
        rng = np.random.default_rng(seed)
        p = rng.choice(case["n"], size=case["tasks"], replace=case["tasks"] > case["n"])
        rows = base[torch.from_numpy(p).to(DEV)].cpu().numpy()
        found = gi.beam_search(rows, case["L"], self_ids=p)
        s["tasks"] = [(int(i), v[0].copy(), v[1].copy()) for i, (_, v, _) in zip(p, found)]
        return s
    if case["beam"]:
        Ls = np.full(case["nq"], case["beam"], np.uint32)
    else:
        Ls = np.array([10, 20, 50, 100, 200], np.uint32)[
            np.random.default_rng(seed).integers(0, 5, case["nq"])]
    if kind == "search":
        s["queries"], s["L"] = q.cpu().numpy(), Ls
        return s
    # device queries: rows zero padded to a multiple of 16 bytes
    per = 16 // ESZ[case["dtype"]]
    dp_ = -(-case["d"] // per) * per
    s["q"] = torch.zeros((case["nq"], dp_), device=DEV, dtype=q.dtype)
    s["q"][:, :case["d"]] = q
    s["L"] = torch.from_numpy(Ls.astype(np.int32)).to(DEV)
    s["Lmax"] = int(Ls.max())
    s["ids"] = torch.zeros((case["nq"], case["k"]), device=DEV, dtype=torch.int32)
    s["dists"] = torch.zeros((case["nq"], case["k"]), device=DEV, dtype=torch.float32)
    s["vis"] = torch.zeros(case["nq"], device=DEV, dtype=torch.int32)
    s["cmps"] = torch.zeros(case["nq"], device=DEV, dtype=torch.int32)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "bsp":
        g = Graph(case["R"], case["n"])
        BSPIndex().bsp_build(s["bp"], g, s["points"], None, s["dp"])
        return g.rows.view(np.int32)
    gi = s["gi"]
    if kind == "build":
        gi.build(case["L"], case["alpha"], max_fraction=case["xita"], knn_mode=case["knn"],
                 two_pass=case["two_pass"], collect_stats=False)
        return s["graph"]
    if kind == "search":
        ids, d, v, c = gi.search(s["queries"], case["k"], s["L"], limit=case["limit"],
                                 degree_limit=case["degree_limit"])
        return ids.view(np.int32), d, v.view(np.int32), c.view(np.int32)
    if kind == "dsearch":
        gi.search_device(s["q"].data_ptr(), case["nq"], s["q"].stride(0) * s["q"].element_size(),
                         s["L"].data_ptr(), s["Lmax"], case["k"], s["ids"].data_ptr(),
                         s["dists"].data_ptr(), limit=case["limit"],
                         degree_limit=case["degree_limit"], vis_ptr=s["vis"].data_ptr(),
                         cmps_ptr=s["cmps"].data_ptr())
        return s["ids"], s["dists"], s["vis"], s["cmps"]
    if kind == "gt":
        ids, d = gi.groundtruth(s["queries"], case["k"])
        return ids.view(np.int32), d
    out = gi.robust_prune(s["tasks"], case["alpha"])
    flat = np.full(case["tasks"] * case["R"], -1, np.int32)  # the lists, one after another
    ids = np.concatenate(out)
    flat[:ids.size] = ids.view(np.int32)
    return np.array([len(o) for o in out], np.int32), flat


# ------------------------------------------------------------------ what a pass needs
def work(case):
    """Bytes and operations of one pass.  A search of beam width L expands about 1.2 L
    nodes (a row of R ids each) and computes about 16 distances per node, each of one row
    of points; a build is one such search per point."""
    kind, d = case["kind"], case["d"]
    row = d * ESZ[case["dtype"]]
    if kind == "gt":
        n, nq = case["n"], case["nq"]
        return {"bytes": n * row + nq * row + nq * case["k"] * 8, "flops": 2.0 * n * nq * d}
    if kind == "prune":
        m = 1.2 * case["L"] + case["R"]
        return {"bytes": case["tasks"] * (m * (row + 8) + case["R"] * 4),
                "flops": case["tasks"] * m * case["R"] * 2.0 * d}
    if kind in ("search", "dsearch"):
        beam = case["beam"] or 76  # the mean of the mixed widths
        beam = min(beam, case["limit"]) if case["limit"] else beam
        deg, n = case["degree_limit"] or case["R"], case["nq"]
    else:
        beam, deg, n = case["L"], case["R"], case["n"] * (2 if case["two_pass"] else 1)
    nodes = 1.2 * beam
    return {"bytes": n * (nodes * 4 * deg + 16 * nodes * row), "flops": n * 16 * nodes * 2.0 * d}


def exact(case, seed):
    """Ground truth distances in 64 bits.  The other outputs are ids, graphs and counts
    (whole numbers), or distances to ids that only a search of the graph gives."""
    if case["kind"] != "gt":
        return None
    base, q = _sets(case, seed)
    l2 = case["metric"] == "l2"
    q = q.double()
    best = None
    step = max(1, int(2e8) // max(1, case["nq"]))
    for s in range(0, case["n"], step):
        b = base[s:s + step].double()
        v = -(q @ b.T)
        if l2:
            v = 2.0 * v
            v += (b * b).sum(1)[None, :]
            v += (q * q).sum(1)[:, None]
        v = v if best is None else torch.cat([best, v], 1)
        best = v.topk(min(case["k"], v.shape[1]), dim=1, largest=False, sorted=True).values
    return None, best
