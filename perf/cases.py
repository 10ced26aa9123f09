"""Performance cases: what users of the engine have it do, through its public entry points.

Every case names an operation (`op`), the index it runs on (type, rows, dimensions, clusters) and
the call's own sizes. Data is synthetic: unit-normalised (or plain) Gaussian mixtures, generated
on the GPU, as in the benchmark's workloads. An index depends on the case alone and is built once
per process, as a serving program keeps one index for many batches; queries, filters and rows to
append come from the seed.

  search        search_device: a batch of GPU-resident queries (serving from a GPU pipeline)
  search_host   search_batch: host queries in, host results out
  single        search: one host query, the reference's own call
  filtered      filtered_search_batch: host queries, one row-id list per query
  requests      Context.search_requests: a continuous-batching step, per-request k / nprobe and
                registered filters
  update        append_batch, search_batch, delete of the same rows: an index under maintenance
  build         build_index from host rows, then save
"""
import math
import os
import tempfile

import numpy as np
import torch

from pdx_b200 import compiled

_CACHE_MAX = 10
_indexes = {}  # index configuration -> (index, registered filter ids), most recent last

# Requests of a serving batch (the benchmark's serving mix).
_REQ_K = (10, 20, 100)
_REQ_NPROBE = (8, 32, 64)
_REQ_FILTERS = 16


def listed():
    big = dict(itype="pdx_tree_u8", n=1_000_000, d=1024, comps=1024, sigma=0.25, unit=True, nlist=1000, nmeso=32)
    return [
        # the headline workload: a large batch against the two-level SQ8 index
        dict(name="tree_u8_batch", op="search", **big, nprobe=32, k=20, nq=10_000),
        # the same index behind the reference's one-query call: latency of an interactive search
        dict(name="tree_u8_single", op="single", **big, nprobe=32, k=20, nq=1),
        # a mid-size host batch of ragged size: an offline job, a web backend that collects queries
        dict(name="tree_u8_host", op="search_host", **big, nprobe=24, k=10, nq=777),
        # the reduced-precision probe option (BF16 tensor-core rotation and centroid scores)
        dict(name="tree_u8_probe_bf16", op="search", **big, nprobe=32, k=20, nq=1024, probe_mode=1),
        # filtered search: selectivities from one in a thousand to one half
        dict(name="tree_u8_filtered", op="filtered", **big, nprobe=32, k=20, nq=16),
        # one step of the serving loop: mixed k, nprobe and registered filters
        dict(name="tree_u8_requests", op="requests", **big, nprobe=64, k=100, nq=512),
        # float32 tree: the operating point without quantisation loss
        dict(name="tree_f32_batch", op="search", itype="pdx_tree_f32", n=200_000, d=768, comps=512, sigma=0.25,
             unit=True, nlist=0, nmeso=0, nprobe=32, k=10, nq=2000),
        # plain IVF, small dimension, not normalised
        dict(name="ivf_f32_batch", op="search", itype="pdx_f32", n=100_000, d=128, comps=256, sigma=0.3,
             unit=False, nlist=316, nmeso=0, nprobe=16, k=10, nq=1000),
        # every cluster visited (nprobe 0): exact search, ground truth
        dict(name="flat_f32_exhaustive", op="search", itype="pdx_f32", n=200_000, d=768, comps=512, sigma=0.2,
             unit=True, nlist=0, nmeso=0, nprobe=0, k=100, nq=300),
        # plain IVF SQ8 with a dimension that is no power of two and a ragged batch
        dict(name="ivf_u8_batch", op="search", itype="pdx_u8", n=150_000, d=200, comps=400, sigma=0.25,
             unit=True, nlist=0, nmeso=0, nprobe=20, k=15, nq=515),
        # rows that come in, are searched beside and are withdrawn again
        dict(name="tree_u8_update", op="update", itype="pdx_tree_u8", n=100_000, d=256, comps=300, sigma=0.25,
             unit=True, nlist=0, nmeso=0, nprobe=16, k=10, nq=64, rows=2048),
        # a build from host rows to a saved index
        dict(name="tree_u8_build", op="build", itype="pdx_tree_u8", n=100_000, d=768, comps=300, sigma=0.25,
             unit=True, nlist=0, nmeso=0, nprobe=0, k=0, nq=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["search", "search", "search", "search_host", "single", "filtered", "requests", "update", "build"])
    itype = rng.choice(["pdx_f32", "pdx_u8", "pdx_tree_f32", "pdx_tree_u8", "pdx_tree_u8"])
    if op == "update":
        itype = rng.choice(["pdx_tree_f32", "pdx_tree_u8"])
    d = 8 * _log_int(rng, 8, 128)
    n = _log_int(rng, 20_000, 300_000)
    if op in ("update", "build"):
        n = min(n, 100_000)
    c = dict(op=op, itype=itype, n=n, d=d, comps=_log_int(rng, 64, 1024), sigma=rng.choice([0.2, 0.25, 0.3]),
             unit=rng.random() < 0.75, nlist=rng.choice([0, 0, max(40, n // 1000)]), nmeso=0,
             nprobe=_log_int(rng, 4, 64), k=rng.choice([1, 5, 10, 20, 37, 100]), nq=0)
    if op == "search":
        c["nq"] = _log_int(rng, 33, 8000)
        if itype == "pdx_f32" and rng.random() < 0.2:
            c.update(nprobe=0, n=min(n, 100_000), nq=_log_int(rng, 33, 300))
        elif d % 16 == 0 and rng.random() < 0.15:
            c["probe_mode"] = rng.choice([1, 2])
    elif op == "search_host":
        c["nq"] = _log_int(rng, 2, 5000)
    elif op == "single":
        c["nq"] = 1
    elif op == "filtered":
        c["nq"] = _log_int(rng, 1, 32)
    elif op == "requests":
        c.update(nq=_log_int(rng, 16, 1024), k=max(_REQ_K), nprobe=max(_REQ_NPROBE))
    elif op == "update":
        c.update(nq=_log_int(rng, 8, 256), rows=_log_int(rng, 64, 4096))
    else:
        c.update(k=0, nprobe=0)
    return c


# ------------------------------------------------------------------------------------- data
def _nlist(case):
    """Clusters of the index (0: the reference's default for n rows below 500,000)."""
    return case["nlist"] or math.ceil(2 * math.sqrt(case["n"]))


def _mixture(case, n, seed):
    """n rows of the case's Gaussian mixture on the GPU; the centres depend on the case alone."""
    d = case["d"]
    g = torch.Generator(device="cuda").manual_seed(1 + d * 31 + case["comps"])
    centres = torch.randn(case["comps"], d, generator=g, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = torch.empty(n, d, device="cuda")
    for s in range(0, n, 1 << 16):
        m = min(1 << 16, n - s)
        label = torch.randint(0, case["comps"], (m,), generator=g, device="cuda")
        x = torch.randn(m, d, generator=g, device="cuda") * case["sigma"] + centres[label]
        out[s:s + m] = x / x.norm(dim=1, keepdim=True) if case["unit"] else x
    return out


def _data(case):
    return _mixture(case, case["n"], 7)


def _queries(case, seed):
    return _mixture(case, case["nq"], 1000 + seed)


def _new_index(case):
    return compiled.PDXIndex(case["itype"], case["d"], seed=11, num_clusters=_nlist(case),
                             num_meso_clusters=case["nmeso"], normalize=case["unit"])


def _build(case):
    ix = _new_index(case)
    ix.build_index(_data(case).cpu().numpy())
    return ix


def _index(case):
    """The program's index, with the filters that a serving program registers."""
    key = tuple((k, case[k]) for k in ("itype", "n", "d", "comps", "sigma", "unit", "nlist", "nmeso"))
    got = _indexes.pop(key, None)
    if got is None:
        while len(_indexes) >= _CACHE_MAX:
            _indexes.pop(next(iter(_indexes)))
        got = (_build(case), [])
    _indexes[key] = got
    return got


def _selection(rng, n):
    """Ascending row ids of one filter: selectivity 0.001 to 0.5, log-uniform."""
    s = math.exp(rng.uniform(math.log(0.001), math.log(0.5)))
    return np.flatnonzero(rng.random(n) < s).astype(np.uint64)


def _filter_rows(case, i):
    return _selection(np.random.default_rng([5, i]), case["n"])


def _requests(case, seed):
    rng = np.random.default_rng([9, seed])
    nq = case["nq"]
    return (rng.choice(_REQ_K, nq).astype(np.uint32), rng.choice(_REQ_NPROBE, nq).astype(np.uint32),
            np.where(rng.random(nq) < 0.5, rng.integers(0, _REQ_FILTERS, nq), -1))


# ------------------------------------------------------------------------------------- passes
def prepare(case, seed):
    op = case["op"]
    s = dict(case=case, op=op, k=case["k"], nq=case["nq"])
    if op == "build":
        s["rows"] = _mixture(case, case["n"], 1000 + seed).cpu().numpy()
        s["path"] = os.path.join(tempfile.gettempdir(), "perf_case_build_%d.pdx" % os.getpid())
        return s
    if op == "update":
        s["ix"] = _build(case)
        s["rows"] = _mixture(case, case["rows"], 5000 + seed).cpu().numpy()
        s["next"] = case["n"]
        s["q"] = _queries(case, seed).cpu().numpy()
        s["ix"].set_nprobe(case["nprobe"])
        return s
    ix, filters = _index(case)
    s["ix"] = ix
    s["nprobe"] = case["nprobe"]
    s["probe_mode"] = case.get("probe_mode", 0)
    q = _queries(case, seed)
    if op in ("search", "requests"):
        s["q"] = q
        s["ids"] = torch.empty(case["nq"], case["k"], dtype=torch.int32, device="cuda")
        s["d"] = torch.empty(case["nq"], case["k"], device="cuda")
        s["cnt"] = torch.empty(case["nq"], dtype=torch.int32, device="cuda")
    else:
        s["q"] = q.cpu().numpy()
    if op == "filtered":
        rng = np.random.default_rng([3, seed])
        s["lists"] = [_selection(rng, case["n"]) for _ in range(case["nq"])]
    if op == "requests":
        if not filters:
            filters.extend(ix.register_filter(_filter_rows(case, i)) for i in range(_REQ_FILTERS))
        k, nprobe, fil = _requests(case, seed)
        table = compiled.request_table(case["nq"])
        table["k"], table["nprobe"] = k, nprobe
        table["filter_id"] = np.where(fil < 0, -1, np.asarray(filters)[np.maximum(fil, 0)])
        s["table"] = table
        s["ctx"] = compiled.Context(ix)
    torch.cuda.synchronize()
    return s


def run(s):
    op, ix = s["op"], s.get("ix")
    if op == "build":
        ix = _new_index(s["case"])
        ix.build_index(s["rows"])
        ix.save(s["path"])
        return {"file": np.fromfile(s["path"], dtype=np.uint8)}
    if op == "update":
        first = s["next"]
        ix.append_batch(first, s["rows"])
        s["next"] = first + len(s["rows"])
        ids, d, cnt = ix.search_batch(s["q"], s["k"])
        for row in range(first, s["next"]):
            ix.delete(row)
        return {"ids": ids.view(np.int32), "distances": d, "counts": cnt.view(np.int32)}
    ix.set_probe_mode(s["probe_mode"])
    if op == "requests":
        s["ctx"].search_requests(s["q"].data_ptr(), s["nq"], s["table"], None, s["k"], s["ids"].data_ptr(),
                                 s["d"].data_ptr(), s["cnt"].data_ptr())
        return {"ids": s["ids"], "distances": s["d"], "counts": s["cnt"]}
    ix.set_nprobe(s["nprobe"])
    if op == "search":
        ix.search_device(s["q"].data_ptr(), s["nq"], s["k"], s["ids"].data_ptr(), s["d"].data_ptr(),
                         s["cnt"].data_ptr())
        return {"ids": s["ids"], "distances": s["d"], "counts": s["cnt"]}
    if op == "single":
        ids, d = ix.search(s["q"][0], s["k"])
        return {"ids": ids.view(np.int32), "distances": d}
    if op == "filtered":
        ids, d, cnt = ix.filtered_search_batch(s["q"], s["k"], s["lists"])
    else:
        ids, d, cnt = ix.search_batch(s["q"], s["k"])
    return {"ids": ids.view(np.int32), "distances": d, "counts": cnt.view(np.int32)}


# ------------------------------------------------------------------------------------- work
def work(case):
    """What a pass cannot do without: queries and results once, the rotation, the centroid probe
    (half of the L1 centroids on a tree), every vector of each query's first cluster, the first 16
    dimensions of the other visited clusters; index bytes at most once per batch."""
    n, d, nq, k = case["n"], case["d"], case["nq"], case["k"]
    nlist = _nlist(case)
    elem = 1 if case["itype"].endswith("u8") else 4
    if case["op"] == "build":
        iters = 11  # assignments of ten k-means updates
        return {"bytes": n * d * (4 + elem) + 4 * d * d, "flops": 2 * n * d * d + 2 * iters * n * nlist * d}
    tree = "tree" in case["itype"]
    size = n / nlist
    nprobe = nlist if case["nprobe"] == 0 else min(case["nprobe"], nlist)
    cents = nlist / 2 + math.sqrt(nlist) if tree and case["op"] != "filtered" else nlist
    started = nlist * (1 - (1 - 1 / nlist) ** nq)
    visited = nlist * (1 - (1 - nprobe / nlist) ** nq)
    dims1 = min(16, d)
    b = nq * d * 4 + nq * k * 8 + nq * 4 + 4 * d * d + cents * d * 4
    b += started * size * d * elem + max(0.0, visited - started) * size * dims1 * elem
    f = 2 * nq * d * d + 3 * nq * cents * d + 3 * nq * size * (d + (nprobe - 1) * dims1)
    if case["op"] == "filtered":
        b += nq * n * 0.08 * 8  # row-id lists, log-uniform selectivity
    if case["op"] == "update":
        b += 2 * case["rows"] * d * (4 + elem)
        f += 2 * case["rows"] * d * d + 3 * case["rows"] * cents * d
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------- exact
def _nearest(q, x, k, allowed=None):
    """Squared distances to the k nearest rows of x in float64, ascending; allowed: [nq, n] mask."""
    q = q.double()
    best = torch.full((len(q), k), float("inf"), dtype=torch.float64, device="cuda")
    step = max(1, min(len(x), (1 << 28) // max(1, len(q))))
    for s in range(0, len(x), step):
        xs = x[s:s + step].double()
        dist = (q * q).sum(1, keepdim=True) - 2.0 * q @ xs.T + (xs * xs).sum(1)[None, :]
        if allowed is not None:
            dist = dist.masked_fill(~allowed[:, s:s + step], float("inf"))
        best = torch.topk(torch.cat([best, dist], 1), k, dim=1, largest=False).values
    return best.clamp(min=0.0)


def _unit64(x):
    return x.double() / x.double().norm(dim=1, keepdim=True)


def exact(case, seed):
    """The true nearest neighbours' squared distances; ids and counts have no such value."""
    op, n, k = case["op"], case["n"], case["k"]
    if op == "build":
        return None
    x, q = _data(case), _queries(case, seed)
    if op == "update":
        x = torch.cat([x, _mixture(case, case["rows"], 5000 + seed)])
    if case["unit"]:
        q = _unit64(q)
    if op == "single":
        return {"ids": None, "distances": _nearest(q, x, k)[0]}
    if op == "filtered":
        rng = np.random.default_rng([3, seed])
        allowed = torch.zeros(case["nq"], n, dtype=torch.bool, device="cuda")
        for i in range(case["nq"]):
            allowed[i, torch.from_numpy(_selection(rng, n).astype(np.int64)).cuda()] = True
        return {"ids": None, "distances": _nearest(q, x, k, allowed), "counts": None}
    if op == "requests":
        kq, _, fil = _requests(case, seed)
        out = torch.empty(case["nq"], k, dtype=torch.float64, device="cuda")
        for f in range(-1, _REQ_FILTERS):
            at = torch.from_numpy(np.flatnonzero(fil == f)).cuda()
            if len(at):
                rows = x if f < 0 else x[torch.from_numpy(_filter_rows(case, f).astype(np.int64)).cuda()]
                out[at] = _nearest(q[at], rows, k)
        past = torch.arange(k)[None, :] >= torch.from_numpy(kq.astype(np.int64))[:, None]
        return {"ids": None, "distances": out.masked_fill(past.cuda(), float("inf")), "counts": None}
    return {"ids": None, "distances": _nearest(q, x, k), "counts": None}
