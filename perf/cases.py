"""Timed cases of the library's main paths, over the range of sizes in which
they are used.

A case is a dict of plain values. `prepare` makes what a program has in hand
before the call (points, a built index, a batch object, queries), `run` is one
call through the public entry points, `work` what that call cannot do without.
Data are seeded Gaussian mixtures of the same shapes as the benchmark's
(uint8: centres in [32, 224], sigma 20; float: centres N(0, 1), sigma 0.3, rows
normalised; int8: the uint8 values shifted by 128), about 4,000 points a
component.

Kinds:
  search      k-NN search through Index.search (host arrays)
  device      k-NN search on device-resident queries (pann_search_device)
  batch       reusable batch with per-query k and beam, exact distances
  tile        reusable batch, low-precision multi-parent tile search
  quantized   one-byte quantized search with float re-rank
  range       greedy range search into a caller's buffer (pann_range_search)
  build       Vamana graph build
  groundtruth exact brute-force top-k
"""
import ctypes
import math

import numpy as np
import torch

import parlayann_b200 as P

U8, I8, F32 = "u8", "i8", "f32"
L2, MIPS = "l2", "mips"
_METRIC = {L2: P.L2, MIPS: P.MIPS}


def listed():
    return [
        # one query at a time, as an interactive caller sends it: latency
        dict(name="search_one", kind="search", dtype=U8, metric=L2, n=100_000, d=128, R=32, bL=64, nq=1, k=10, L=20),
        # the small uint8 configuration: 1,000 queries at a mid beam
        dict(name="search_u8", kind="search", dtype=U8, metric=L2, n=100_000, d=128, R=32, bL=64, nq=1000, k=10, L=50),
        # the benchmark's workload: 10,000 resident float queries on 1M points
        dict(name="search_f32", kind="device", dtype=F32, metric=L2, n=1_000_000, d=96, R=64, bL=64, nq=10_000, k=10,
             L=45),
        # high recall, many neighbours, inner product, sizes that divide nothing
        dict(name="search_i8_mips", kind="search", dtype=I8, metric=MIPS, n=60_001, d=100, R=48, bL=64, nq=777, k=100,
             L=150),
        # callers with different needs in one batch: k in {1, 10, 100}, beam in [k, 4k]
        dict(name="batch_uneven", kind="batch", dtype=F32, metric=L2, n=200_000, d=96, R=64, bL=64, nq=4000, k=100,
             L=400),
        # the throughput form: FP8 tile search at recall about 0.95
        dict(name="tile_fp8", kind="tile", dtype=F32, metric=L2, n=500_000, d=96, R=64, bL=64, nq=10_000, k=10, L=45,
             prec="fp8", parents=3),
        # the reference's own mixed precision: one-byte traversal, float re-rank
        dict(name="quantized", kind="quantized", dtype=F32, metric=L2, n=200_000, d=96, R=64, bL=64, nq=4096, k=10,
             L=45),
        # every point within a radius (the 1 % quantile of the distances): clustering, near duplicates
        dict(name="range_f32", kind="range", dtype=F32, metric=L2, n=200_000, d=96, R=64, bL=64, nq=200, beam=10,
             quantile=0.01),
        # index construction, small uint8 configuration: two passes, R 32, L 64
        dict(name="build_u8", kind="build", dtype=U8, metric=L2, n=100_000, d=128, R=32, bL=64, passes=2),
        # index construction with the benchmark's parameters: R 64, L 128
        dict(name="build_f32", kind="build", dtype=F32, metric=L2, n=100_000, d=96, R=64, bL=128, passes=2),
        # exact answers to measure recall against, byte vectors
        dict(name="groundtruth_u8", kind="groundtruth", dtype=U8, metric=L2, n=100_000, d=128, nq=1000, k=100),
        # exact answers at the benchmark's size
        dict(name="groundtruth_f32", kind="groundtruth", dtype=F32, metric=L2, n=1_000_000, d=96, nq=10_000, k=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "device", "batch", "tile", "quantized", "range", "build", "groundtruth"])
    dtype = rng.choice([U8, I8, F32, F32])
    metric = rng.choice([L2, L2, MIPS])
    if kind in ("tile", "quantized"):
        dtype = F32
    c = dict(kind=kind, dtype=dtype, metric=metric, n=_log(rng, 5_000, 300_000), d=_log(rng, 24, 256))
    if kind == "groundtruth":
        c.update(nq=_log(rng, 10, 5_000), k=rng.choice([1, 10, 20, 100]))
        return c
    c.update(R=rng.choice([24, 32, 48, 64]), bL=rng.choice([48, 64, 96]))
    if kind == "build":
        c.update(n=_log(rng, 5_000, 60_000), passes=rng.choice([1, 2]))
        return c
    if kind == "range":
        c.update(metric=L2, nq=_log(rng, 10, 400), beam=rng.choice([10, 20, 50]), quantile=rng.choice([0.001, 0.003, 0.01]))
        return c
    c.update(nq=_log(rng, 1, 8_000))
    if kind == "batch":
        c.update(nq=_log(rng, 50, 4_000), k=rng.choice([10, 50, 100]))
        c["L"] = c["k"] * rng.randint(2, 4)
        return c
    c["k"] = rng.choice([1, 10, 10, 50])
    c["L"] = c["k"] + _log(rng, 10, 150)
    if kind == "tile":
        c["d"] += c["d"] % 2  # pairs of values are scored together
        c.update(prec=rng.choice(["bf16", "fp8"]), parents=rng.choice([2, 3]))
    return c


# ---------------------------------------------------------------- inputs


def _mixture(c, seed, rows, stream, gen_rows=1 << 18):
    """`rows` points of the case's mixture on the GPU (the centres depend on the seed alone)."""
    comps = max(8, c["n"] // 4000)
    g = torch.Generator("cuda").manual_seed(int(seed) * 16 + 1)
    if c["dtype"] == F32:
        cen = torch.randn((comps, c["d"]), generator=g, device="cuda")
    else:
        cen = 32 + 192 * torch.rand((comps, c["d"]), generator=g, device="cuda")
    g = torch.Generator("cuda").manual_seed(int(seed) * 16 + 2 + stream)
    out = []
    for at in range(0, rows, gen_rows):
        m = min(gen_rows, rows - at)
        x = cen[torch.randint(comps, (m,), generator=g, device="cuda")]
        noise = torch.randn((m, c["d"]), generator=g, device="cuda")
        if c["dtype"] == F32:
            x = x + 0.3 * noise
            out.append(x / x.square().sum(1, keepdim=True).sqrt())
        else:
            x = (x + 20 * noise).round().clamp(0, 255)
            out.append(x.to(torch.uint8) if c["dtype"] == U8 else (x - 128).to(torch.int8))
    return torch.cat(out)


def _radius(base, q, quantile):
    """The quantile of the squared distances of the queries to a sample of the points."""
    a, b = q[:64].double(), base[:: max(1, len(base) // 4096)].double()
    dd = (a[:, None, :] - b[None, :, :]).square().sum(2).flatten()
    return float("%.3g" % float(torch.sort(dd).values[int(quantile * len(dd))]))


def prepare(case, seed):
    c = case
    s = dict(case=c)
    base = _mixture(c, seed, c["n"], 0)
    q = _mixture(c, seed, c["nq"], 1) if "nq" in c else None
    idx = P.Index(base.cpu().numpy(), c.get("R", 32), _METRIC[c["metric"]])
    s["idx"] = idx
    if c["kind"] in ("build", "groundtruth"):
        s["q"] = q.cpu().numpy() if q is not None else None
        return s
    idx.build(L=c["bL"], alpha=1.2 if c["metric"] == L2 else 1.0, num_passes=1)
    if c["kind"] == "device":
        s["q"] = q.contiguous()
        s["ids"] = torch.empty((c["nq"], c["k"]), dtype=torch.int32, device="cuda")
        s["dists"] = torch.empty((c["nq"], c["k"]), dtype=torch.float32, device="cuda")
        s["visited"] = torch.empty(c["nq"], dtype=torch.int32, device="cuda")
        s["cmps"] = torch.empty(c["nq"], dtype=torch.int32, device="cuda")
        s["qp"] = P.QueryParams(c["k"], c["L"], c["n"], c["R"], 0.125)
        s["start"] = np.zeros(1, np.uint32)
        return s
    s["q"] = q.cpu().numpy()
    if c["kind"] == "batch":
        r = np.random.default_rng(seed)
        k = r.choice([x for x in (1, 10, 100) if x <= c["k"]], c["nq"]).astype(np.uint32)
        k[0] = c["k"]
        s["k"] = k
        s["beam"] = (k * r.uniform(1.0, c["L"] / c["k"], c["nq"])).astype(np.uint32)
        s["batch"] = idx.batch(c["nq"], c["k"], c["L"])
    elif c["kind"] == "tile":
        prec = P.PREC_FP8 if c["prec"] == "fp8" else P.PREC_BF16
        idx.set_precision(prec)
        s["batch"] = idx.batch(c["nq"], c["k"], c["L"], precision=prec, parents=c["parents"])
    elif c["kind"] == "quantized":
        idx.set_quantized()
    elif c["kind"] == "range":
        # the caller's answer buffer: 8 times the answers the quantile stands for
        cap = int(8 * c["nq"] * c["n"] * c["quantile"]) + 1024
        s["rp"] = P.RangeParams(c["beam"], P.RANGE_GREEDY, _radius(base, q, c["quantile"]), 0.0, 0)
        s["ids"] = np.zeros(cap, np.uint32)
        s["offsets"] = np.zeros(c["nq"] + 1, np.uint64)
        s["visited"], s["cmps"], s["flags"] = (np.zeros(c["nq"], np.uint32) for _ in range(3))
    return s


# ---------------------------------------------------------------- one pass


def _answer(r):
    return dict(ids=r.ids, dists=r.dists, visited=r.visited, cmps=r.cmps)


def run(state):
    c, idx = state["case"], state["idx"]
    kind = c["kind"]
    if kind == "search":
        return _answer(idx.search(state["q"], c["k"], c["L"], allow_short=True))
    if kind == "device":
        q, ids, dists, vis, cmps = (state[x] for x in ("q", "ids", "dists", "visited", "cmps"))
        start = state["start"]
        rc = P.lib().pann_search_device(idx.handle, q.data_ptr(), c["nq"], ctypes.byref(state["qp"]),
                                        start.ctypes.data, 1, ids.data_ptr(), dists.data_ptr(), vis.data_ptr(),
                                        cmps.data_ptr(), None, torch.cuda.current_stream().cuda_stream)
        if rc:
            raise P.PannError(rc, P.lib().pann_last_error().decode())
        return dict(ids=ids, dists=dists, visited=vis, cmps=cmps)
    if kind == "batch":
        return _answer(state["batch"].run(state["q"], state["k"], state["beam"], allow_short=True))
    if kind == "tile":
        return _answer(state["batch"].run(state["q"], c["k"], c["L"], allow_short=True))
    if kind == "quantized":
        return _answer(idx.search_quantized(state["q"], c["k"], c["L"]))
    if kind == "range":
        q, ids, offs, vis, cmps, flags = (state[x] for x in ("q", "ids", "offsets", "visited", "cmps", "flags"))
        rc = P.lib().pann_range_search(idx.handle, q.ctypes.data, c["nq"], ctypes.byref(state["rp"]), 0,
                                       offs.ctypes.data, ids.ctypes.data, len(ids), vis.ctypes.data, cmps.ctypes.data,
                                       flags.ctypes.data)
        if rc:
            raise P.PannError(rc, P.lib().pann_last_error().decode())
        return dict(ids=ids, offsets=offs.view(np.int64), visited=vis, cmps=cmps)
    if kind == "build":
        st = idx.build(L=c["bL"], alpha=1.2 if c["metric"] == L2 else 1.0, num_passes=c["passes"])
        return dict(graph=idx.get_graph(), dist_cmps=int(st.dist_cmps), visited=int(st.visited_total))
    ids, dists = idx.groundtruth(state["q"], c["k"])
    return dict(ids=ids, dists=dists)


# ---------------------------------------------------------------- what a pass needs


def _search_bytes(c, row, nq, L, k):
    """Adjacency rows of the visited nodes (about 1.3 a beam entry), the rows
    scored (about half of their neighbours are new), queries and answers."""
    visits, deg = 1.3 * L, 0.8 * c["R"]
    return nq * (4 * visits * (1 + deg) + 0.5 * visits * deg * row + row + 8 * k + 8), nq * visits * 0.5 * deg


def work(case):
    c = case
    row = c["d"] * (4 if c["dtype"] == F32 else 1)
    kind = c["kind"]
    if kind == "groundtruth":
        return dict(bytes=(c["n"] + c["nq"]) * row + 12 * c["nq"] * c["k"], flops=2.0 * c["nq"] * c["n"] * c["d"])
    if kind == "build":
        # an insertion search and one robustPrune a point and pass, the reverse edges' prunes
        b, rows = _search_bytes(c, row, c["n"], c["bL"], 0)
        prune = c["n"] * (1.3 * c["bL"] + 2 * c["R"])
        return dict(bytes=c["passes"] * (b + prune * row) + 4 * c["n"] * c["R"],
                    flops=c["passes"] * 3.0 * c["d"] * (rows + prune * c["R"] / 2))
    if kind == "range":
        answers = c["nq"] * c["n"] * c["quantile"]
        b, rows = _search_bytes(c, row, c["nq"], c["beam"], 0)
        return dict(bytes=b + answers * (4 * c["R"] + row + 4), flops=3.0 * c["d"] * (rows + answers))
    L = c["L"] / 2 if kind == "batch" else c["L"]
    if kind == "batch":
        L *= 0.4  # the mean over k in {1, 10, 100}
    lp = {"tile": 1 if c.get("prec") == "fp8" else 2, "quantized": 1}.get(kind)
    b, rows = _search_bytes(c, c["d"] * lp if lp else row, c["nq"], L, c["k"])
    return dict(bytes=b, flops=3.0 * c["d"] * rows)


def exact(case, seed):
    """The exact top-k and its distances for the groundtruth cases; the other
    answers depend on the order of an approximate search and have no such value."""
    c = case
    if c["kind"] != "groundtruth":
        return None
    base, q = _mixture(c, seed, c["n"], 0).double(), _mixture(c, seed, c["nq"], 1).double()
    k = min(c["k"], c["n"])
    more = min(2 * k + 16, c["n"])
    bn = base.square().sum(1)
    ids, dists = [], []
    step = max(1, (1 << 28) // c["n"])
    for at in range(0, c["nq"], step):
        a = q[at:at + step]
        dd = -(a @ base.T)
        if c["metric"] == L2:
            dd = 2 * dd + bn
        near = torch.topk(dd, more, dim=1, largest=False).indices.sort(dim=1).values
        rows = base[near]
        dd = (rows - a[:, None, :]).square().sum(2) if c["metric"] == L2 else -(rows * a[:, None, :]).sum(2)
        best = torch.sort(dd, dim=1, stable=True)
        ids.append(near.gather(1, best.indices[:, :k]))
        dists.append(best.values[:, :k])
    return dict(ids=torch.cat(ids).cpu().numpy().astype(np.uint32), dists=torch.cat(dists).cpu().numpy())
