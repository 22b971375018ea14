"""Workloads of the kNN-graph engine, each one pass through a public entry point.

A user of the engine clusters a set of embeddings: the rows (f32, int8 or
packed bits) become a kNN graph, the graph a fuzzy simplicial set, label
propagation and node embedding lay it out in a few dimensions, and a minimum
spanning tree of the layout is condensed into clusters.  The cases are those
calls over the sizes of the repository's benchmark configurations, tests and
serving stream (500 to 1,000,000 rows, 64 to 1,024 features), ragged sizes
included.  Rows are drawn as the benchmark draws them (clustered, unit
length), and in one case without clusters.

  listed()            the cases
  draw(rng)           another case of the same ranges
  prepare(case, seed) inputs on the GPU
  run(state)          one pass and its outputs
  work(case)          bytes and operations a pass cannot do without
  exact(case, seed)   the outputs in 64 bits, where they have such a value
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "evoc-rs_b200"))

import evoc  # noqa: E402
from evoc import _lib  # noqa: E402
from evoc.boruvka import parallel_boruvka_device  # noqa: E402
from evoc.label_prop import label_propagation_init_device, node_embedding_device  # noqa: E402

DTYPES = {"f32": _lib.DTYPE_F32, "i8": _lib.DTYPE_I8, "bits": _lib.DTYPE_U8}


def listed():
    return [
        # the quickstart set (the benchmark's 2,000 x 128 blobs): every launch and read-back counts
        {"name": "knn_f32_2k_128", "kind": "knn", "dtype": "f32", "n": 2000, "d": 128, "k": 15, "clusters": 10,
         "spread": 0.3, "zipf": 0.0},
        # an ordinary small collection, ragged in n: text or image embeddings of a few thousand documents per topic
        {"name": "knn_f32_20k_384", "kind": "knn", "dtype": "f32", "n": 20011, "d": 384, "k": 15, "clusters": 50,
         "spread": 0.4, "zipf": 0.0},
        # rows without cluster structure, a feature count that is no multiple of any tile
        {"name": "knn_f32_50k_200_flat", "kind": "knn", "dtype": "f32", "n": 50000, "d": 200, "k": 15, "clusters": 0,
         "spread": 1.0, "zipf": 0.0},
        # the largest request of the serving stream
        {"name": "knn_f32_200k_768", "kind": "knn", "dtype": "f32", "n": 200000, "d": 768, "k": 30, "clusters": 200,
         "spread": 0.5, "zipf": 1.1},
        # the headline benchmark
        {"name": "knn_f32_1m_768", "kind": "knn", "dtype": "f32", "n": 1000000, "d": 768, "k": 30, "clusters": 200,
         "spread": 0.5, "zipf": 1.1},
        # quantised embeddings (a quarter of the benchmark's int8 set), exact integer ranking
        {"name": "knn_i8_500k_384", "kind": "knn", "dtype": "i8", "n": 500000, "d": 384, "k": 15, "clusters": 100,
         "spread": 0.25, "zipf": 0.0},
        # binary embeddings, Jaccard ranking (the benchmark's bit rows at a sixteenth of its row count)
        {"name": "knn_bits_250k_1024", "kind": "knn", "dtype": "bits", "n": 250000, "d": 1024, "k": 15,
         "clusters": 500, "spread": 0.05, "zipf": 0.0},
        # many small graphs in one call: the serving loop under backlog
        {"name": "batch_f32_64x384", "kind": "batch", "dtype": "f32", "jobs": 64, "n_lo": 500, "n_hi": 8000, "d": 384,
         "k": 15, "clusters": 20, "spread": 0.3, "zipf": 0.0},
        # the fuzzy simplicial set of a kNN graph: the step after every kNN call
        {"name": "fuzzy_300k_30", "kind": "fuzzy", "n": 300000, "d": 64, "k": 30, "clusters": 200, "spread": 0.5,
         "zipf": 1.1},
        # the label-propagation init of that graph
        {"name": "lpinit_200k_256", "kind": "lpinit", "n": 200000, "d": 256, "k": 15, "clusters": 200, "spread": 0.5,
         "zipf": 1.1, "components": 7},
        # the node embedding from that init, reproducible epochs
        {"name": "embed_100k_15", "kind": "embed", "n": 100000, "d": 64, "k": 15, "clusters": 100, "spread": 0.5,
         "zipf": 1.1, "components": 5, "epochs": 50},
        # the minimum spanning tree of an embedding with its core distances
        {"name": "mst_300k_7", "kind": "mst", "n": 300000, "d": 7, "clusters": 40, "min_samples": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["knn_f32", "knn_f32", "knn_f32", "knn_i8", "knn_i8", "knn_bits", "knn_bits", "batch", "fuzzy",
                       "lpinit", "embed", "mst"])
    mix = {"clusters": _log_int(rng, 5, 500), "spread": round(rng.uniform(0.2, 0.9), 3),
           "zipf": rng.choice([0.0, 1.1])}
    if kind.startswith("knn_"):
        dtype = kind[4:]
        d = 8 * rng.randint(8, 128) if dtype == "bits" else rng.randint(64, 1024)
        k = rng.randint(5, 40)
        # an exhaustive search costs n * n * d; the largest listed case has 7.7e14
        n = _log_int(rng, 500, min(600000, int(math.sqrt(1.5e14 / d))))
        if dtype == "bits":
            mix["spread"], mix["zipf"] = round(rng.uniform(0.02, 0.1), 3), 0.0
        elif rng.random() < 0.15:
            mix["clusters"] = 0
        return {"kind": "knn", "dtype": dtype, "n": n, "d": d, "k": k, **mix}
    if kind == "batch":
        lo = _log_int(rng, 200, 2000)
        return {"kind": "batch", "dtype": rng.choice(["f32", "i8"]), "jobs": rng.randint(4, 96), "n_lo": lo,
                "n_hi": 8 * lo, "d": rng.randint(64, 768), "k": rng.randint(5, 30), **mix}
    n = _log_int(rng, 2000, 400000)
    if kind == "fuzzy":
        return {"kind": "fuzzy", "n": n, "d": 64, "k": rng.randint(5, 40), **mix}
    if kind == "lpinit":
        return {"kind": "lpinit", "n": min(n, 250000), "d": rng.randint(64, 400), "k": rng.randint(10, 30),
                "components": rng.randint(4, 15), **mix}
    if kind == "embed":
        return {"kind": "embed", "n": min(n, 150000), "d": 64, "k": rng.randint(10, 30),
                "components": rng.randint(2, 15), "epochs": rng.randint(20, 60), **mix}
    return {"kind": "mst", "n": n, "d": rng.randint(4, 15), "clusters": rng.randint(5, 60),
            "min_samples": rng.randint(2, 12)}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _labels(n, clusters, zipf, g):
    if zipf <= 0.0:
        return torch.randint(0, clusters, (n,), generator=g, device="cuda")
    w = torch.arange(1, clusters + 1, device="cuda", dtype=torch.float64) ** -zipf
    edges = torch.cumsum(w / w.sum(), 0)
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    return torch.searchsorted(edges, u).clamp_(max=clusters - 1)


def _unit_rows(n, d, clusters, spread, zipf, g):
    """Unit f32 rows and their clusters: normal centres plus noise whose size differs by cluster
    and feature (0.2 to 1 times `spread`), in random order; without clusters, normal rows."""
    x = torch.empty(n, d, device="cuda")
    step = 131072
    lab = torch.zeros(n, dtype=torch.int64, device="cuda")
    if clusters:
        centres = torch.randn(clusters, d, generator=g, device="cuda")
        sigma = (0.2 + 0.8 * torch.rand(clusters, d, generator=g, device="cuda")) * spread
        lab = _labels(n, clusters, zipf, g)
    for s in range(0, n, step):
        m = min(step, n - s)
        v = torch.randn(m, d, generator=g, device="cuda")
        if clusters:
            v = centres[lab[s:s + m]] + sigma[lab[s:s + m]] * v
        x[s:s + m] = v / v.norm(dim=1, keepdim=True)
    return x, lab


def _bit_rows(n, bits, clusters, flip, g):
    """Packed bit rows: each copies one of `clusters` prototypes (a tenth of the bits set) and
    flips each bit with probability `flip`."""
    protos = torch.rand(clusters, bits, generator=g, device="cuda") < 0.1
    lab = torch.randint(0, clusters, (n,), generator=g, device="cuda")
    place = (2 ** torch.arange(7, -1, -1, device="cuda")).to(torch.int32)
    out = torch.empty(n, bits // 8, dtype=torch.uint8, device="cuda")
    step = 131072
    for s in range(0, n, step):
        lb = lab[s:s + step]
        rows = protos[lb] ^ (torch.rand(len(lb), bits, generator=g, device="cuda") < flip)
        out[s:s + step] = (rows.view(len(lb), -1, 8).to(torch.int32) * place).sum(-1).to(torch.uint8)
    return out


def _rows(case, n, g):
    if case["dtype"] == "bits":
        return _bit_rows(n, case["d"], case["clusters"], case["spread"], g)
    x, _ = _unit_rows(n, case["d"], case["clusters"], case["spread"], case["zipf"], g)
    if case["dtype"] == "i8":
        x = torch.clamp(torch.round(127.0 * x), -127, 127).to(torch.int8)
    return x


def _knn_into(x, dtype, k, idx, dist):
    evoc.knn_graph_device(x.data_ptr(), DTYPES[dtype], x.shape[0], x.shape[1], k, idx.data_ptr(), dist.data_ptr())


def _knn_outputs(n, k):
    return (torch.empty(n, k, dtype=torch.int32, device="cuda"),
            torch.empty(n, k, dtype=torch.float32, device="cuda"))


def _k_eff(n, k):
    return max(1, min(k, n - 1))


def _ready():
    torch.cuda.current_stream().synchronize()  # the library runs on its own stream


def _fuzzy_into(s):
    ctx = _lib.context(0)
    p = ctypes.c_void_p
    nnz = ctypes.c_int64(0)
    n, k = s["idx"].shape
    st = _lib.lib().evoc_gpu_fuzzy_graph(
        ctx.h, p(s["idx"].data_ptr()), p(s["dist"].data_ptr()), n, k, float(k), 1, 1, p(s["sigma"].data_ptr()),
        p(s["rho"].data_ptr()), p(s["indptr"].data_ptr()), p(s["indices"].data_ptr()), p(s["data"].data_ptr()),
        2 * n * k, ctypes.byref(nnz))
    if st != 0:
        raise RuntimeError(ctx.last_error())


def _knn_state(case, g):
    """A kNN graph as a user holds it (row index, -log2 of the cosine, the row itself first):
    neighbours are searched within groups of 2,000 rows, cluster by cluster."""
    n, k, size = case["n"], _k_eff(case["n"], case["k"]), min(2000, case["n"])
    x, lab = _unit_rows(n, case["d"], case["clusters"], case["spread"], case["zipf"], g)
    by_cluster = torch.argsort(lab, stable=True)
    idx, dist = _knn_outputs(n, k)
    for s in range(0, n, size):
        a = min(s, n - size)
        ids = by_cluster[a:a + size]
        sim = x[ids] @ x[ids].T
        sim.fill_diagonal_(2.0)
        best, at = torch.sort(sim, dim=1, descending=True, stable=True)
        best, at = best[:, :k], at[:, :k]
        idx[ids] = ids[at].to(torch.int32)
        dist[ids] = torch.clamp(-torch.log2(torch.clamp(best, 1e-30, 1.0)), min=0.0)
    return x, {"idx": idx, "dist": dist}


def _fuzzy_outputs(n, k):
    return {"sigma": torch.empty(n, device="cuda"), "rho": torch.empty(n, device="cuda"),
            "indptr": torch.empty(n + 1, dtype=torch.int64, device="cuda"),
            "indices": torch.zeros(2 * n * k, dtype=torch.int32, device="cuda"),
            "data": torch.zeros(2 * n * k, device="cuda")}


def _batch_sizes(case, seed):
    rng = np.random.RandomState(seed)
    u = rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"]), case["jobs"])
    return [int(v) for v in np.exp(u)]


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    s = {"case": case, "seed": seed}
    if kind == "knn":
        s["x"] = _rows(case, case["n"], g)
        s["k"] = _k_eff(case["n"], case["k"])
        s["idx"], s["dist"] = _knn_outputs(case["n"], s["k"])
    elif kind == "batch":
        # all requests' rows and outputs in one allocation each, as a server's pool holds them;
        # the sizes belong to the case, the rows to the seed
        s["ns"] = _batch_sizes(case, case["jobs"])
        s["xs"] = [_rows(case, n, g) for n in s["ns"]]
        s["ks"] = [_k_eff(n, case["k"]) for n in s["ns"]]
        ends = np.cumsum([n * k for n, k in zip(s["ns"], s["ks"])])
        s["starts"] = [0] + [int(e) for e in ends[:-1]]
        s["idx"], s["dist"] = _knn_outputs(int(ends[-1]), 1)
    elif kind == "mst":
        centres = torch.randn(case["clusters"], case["d"], generator=g, device="cuda")
        lab = torch.randint(0, case["clusters"], (case["n"],), generator=g, device="cuda")
        s["x"] = (centres[lab] + 0.15 * torch.randn(case["n"], case["d"], generator=g, device="cuda")).contiguous()
        s["edges"] = torch.zeros(case["n"] - 1, 3, device="cuda")
        s["core"] = torch.zeros(case["n"], device="cuda")
    else:
        s["x"], graph = _knn_state(case, g)
        if kind == "fuzzy":
            s.update(graph)
            s.update(_fuzzy_outputs(*graph["idx"].shape))
        else:
            f = _fuzzy_graph(graph["idx"], graph["dist"])
            s["indptr"], s["indices"], s["data"] = f["indptr"], f["indices"], f["data"].float()
            s["out"] = torch.empty(case["n"], case["components"], device="cuda")
            if kind == "embed":
                s["init"] = 0.5 * torch.randn(case["n"], case["components"], generator=g, device="cuda")
    _ready()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "knn":
        _knn_into(s["x"], case["dtype"], s["k"], s["idx"], s["dist"])
        return {"indices": s["idx"], "distances": s["dist"]}
    if kind == "batch":
        pi, pd = s["idx"].data_ptr(), s["dist"].data_ptr()
        evoc.knn_graph_batch_device([x.data_ptr() for x in s["xs"]], DTYPES[case["dtype"]], s["ns"],
                                    [case["d"]] * len(s["ns"]), case["k"], [pi + 4 * a for a in s["starts"]],
                                    [pd + 4 * a for a in s["starts"]])
        return {"indices": s["idx"], "distances": s["dist"]}
    if kind == "fuzzy":
        _fuzzy_into(s)  # indices and data hold indptr[n] entries, zeros past them
        return {"sigma": s["sigma"], "rho": s["rho"], "indptr": s["indptr"], "indices": s["indices"],
                "data": s["data"]}
    if kind == "lpinit":
        rs = np.random.RandomState(s["seed"] % 2**31)
        label_propagation_init_device(s["indptr"].data_ptr(), s["indices"].data_ptr(), s["data"].data_ptr(),
                                      case["n"], s["x"].data_ptr(), case["d"], s["out"].data_ptr(), rs,
                                      approx_n_parts=min(8000, max(256, case["n"] // 32)),
                                      n_components=case["components"])
        return {"embedding": s["out"], "next_draw": int(rs.randint(2**31 - 1))}
    if kind == "embed":
        rs = np.random.RandomState(s["seed"] % 2**31)
        node_embedding_device(s["indptr"].data_ptr(), s["indices"].data_ptr(), s["data"].data_ptr(), case["n"],
                              case["components"], case["epochs"], s["init"].data_ptr(), s["out"].data_ptr(), rs)
        return {"embedding": s["out"], "next_draw": int(rs.randint(2**31 - 1))}
    parallel_boruvka_device(s["x"].data_ptr(), case["n"], case["d"], case["min_samples"], s["edges"].data_ptr(),
                            s["core"].data_ptr())
    # the hierarchy is built from the edges by ascending length; which of the pairs at one length
    # an edge joins is open (mutual reachability ties are common), the lengths are not
    s["edges"] = s["edges"][torch.argsort(s["edges"][:, 2])]
    return {"core": s["core"], "lengths": s["edges"][:, 2]}


def _row_bytes(case):
    return {"f32": 4 * case.get("d", 0), "i8": case.get("d", 0), "bits": case.get("d", 0) // 8}[
        case.get("dtype", "f32")]


def work(case):
    """Inputs read once and outputs written once.  Operations: of a search, one distance per
    neighbour it reports (an exhaustive one computes n per row, but which of them a search can
    leave out depends on the rows); of the graph steps, a few per edge."""
    kind = case["kind"]
    if kind in ("knn", "batch"):
        ns = [case["n"]] if kind == "knn" else _batch_sizes(case, case["jobs"])
        entries = sum(n * _k_eff(n, case["k"]) for n in ns)
        return {"bytes": sum(ns) * _row_bytes(case) + 8 * entries, "flops": 2 * entries * case["d"]}
    n = case["n"]
    if kind == "mst":
        return {"bytes": 4 * n * case["d"] + 16 * n, "flops": 3 * n * case["d"] * (case["min_samples"] + 1)}
    nk = n * case["k"]
    if kind == "fuzzy":
        return {"bytes": 8 * nk + 8 * int(1.6 * nk) + 16 * n, "flops": 10 * nk}
    graph = 8 * n + 8 * int(1.6 * nk)
    if kind == "lpinit":
        return {"bytes": graph + 4 * n * case["d"] + 4 * n * case["components"], "flops": n * case["d"]}
    return {"bytes": graph + 8 * n * case["components"],
            "flops": case["epochs"] * int(1.6 * nk) * 8 * case["components"]}


def _exact_distances(x, dtype, k):
    """The k smallest distances of every row, ascending, in 64 bits: the row itself counts with
    dissimilarity -1."""
    n = x.shape[0]
    if dtype == "bits":
        place = 2 ** torch.arange(7, -1, -1, device="cuda", dtype=torch.uint8)
        v = ((x[:, :, None] & place) != 0).reshape(n, -1).double()
        size = v.sum(1)
    else:
        v = x.double()
    out = torch.empty(n, k, dtype=torch.float64, device="cuda")
    step = max(1, min(n, int(2e9 / (8 * n))))
    for s in range(0, n, step):
        q = v[s:s + step]
        sim = q @ v.T
        if dtype == "bits":
            union = size[s:s + step, None] + size[None, :] - sim
            sim = torch.where(union > 0, sim / union, torch.zeros_like(sim))
        at = torch.arange(len(q), device="cuda")
        sim[at, at + s] = 1.0
        best = torch.topk(sim, k, dim=1).values
        if dtype == "i8":
            dist = torch.where(best > 0, 1.0 / best, torch.zeros_like(best))
        else:
            dist = torch.where(best > 0, torch.clamp(-torch.log2(best), min=0.0), torch.zeros_like(best))
        out[s:s + step] = dist
    return out


def _fuzzy_graph(idx, dist):
    """The fuzzy simplicial set in 64 bits: 64 steps of bisection on sigma, memberships, then
    a + b - a b as CSR with sorted columns."""
    dist = dist.double()
    n, k = dist.shape
    pos = dist > 0
    first = pos.double().argmax(1)
    rho = torch.where(pos.any(1), dist.gather(1, first[:, None])[:, 0], torch.zeros_like(dist[:, 0]))
    d = dist[:, 1:] - rho[:, None]
    target, tol = math.log2(float(k)), float(np.float32(1e-5))
    lo, hi, mid = torch.zeros_like(rho), torch.full_like(rho, math.inf), torch.ones_like(rho)
    live = torch.ones(n, dtype=torch.bool, device="cuda")
    for _ in range(64):
        ps = torch.where(d > 0, torch.exp(-(d / mid[:, None])), torch.ones_like(d)).sum(1)
        live &= (ps - target).abs() >= tol
        big, small = live & (ps > target), live & ~(ps > target)
        hi, lo = torch.where(big, mid, hi), torch.where(small, mid, lo)
        step = torch.where(torch.isinf(hi), mid * 2, (lo + hi) / 2)
        mid = torch.where(live, step, mid)
    floor = float(np.float32(1e-3))
    sigma = torch.maximum(mid, floor * torch.where(rho > 0, dist.mean(1), dist.mean().expand(n)))
    rows = torch.arange(n, device="cuda")[:, None].expand(n, k)
    dr = dist - rho[:, None]
    w = torch.where((dr <= 0) | (sigma[:, None] == 0), torch.ones_like(dr), torch.exp(-(dr / sigma[:, None])))
    keep = (idx >= 0) & (idx != rows) & (w.float() > 0)
    i, j, w = rows[keep], idx[keep].long(), w[keep]
    key, order = torch.sort(torch.cat([i * n + j, j * n + i]), stable=True)
    val = torch.cat([w, w])[order]
    twin = torch.zeros_like(key, dtype=torch.bool)
    twin[1:] = key[1:] == key[:-1]
    other = torch.zeros_like(val)
    other[:-1] = torch.where(twin[1:], val[1:], other[1:])
    key, val = key[~twin], (val + other - val * other)[~twin]
    counts = torch.bincount(key // n, minlength=n)
    indptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    indptr[1:] = torch.cumsum(counts, 0)
    return {"sigma": sigma, "rho": rho, "indptr": indptr, "indices": (key % n).to(torch.int32), "data": val}


def exact(case, seed):
    kind = case["kind"]
    if kind == "knn":
        if 2.0 * case["n"] ** 2 * case["d"] > 1.3e14:
            return None  # over 20 seconds in 64 bits
        x = _rows(case, case["n"], _generator(seed))
        return {"indices": None, "distances": _exact_distances(x, case["dtype"], _k_eff(case["n"], case["k"]))}
    if kind == "batch":
        g = _generator(seed)
        got = []
        for n in _batch_sizes(case, case["jobs"]):
            got.append(_exact_distances(_rows(case, n, g), case["dtype"], _k_eff(n, case["k"])).reshape(-1, 1))
        return {"indices": None, "distances": torch.cat(got)}
    if kind == "fuzzy":
        s = prepare(case, seed)
        f = _fuzzy_graph(s["idx"], s["dist"])
        data = torch.zeros(len(s["data"]), dtype=torch.float64, device="cuda")
        data[:len(f["data"])] = f["data"]
        return {"sigma": f["sigma"], "rho": f["rho"], "indptr": None, "indices": None, "data": data}
    if kind == "mst" and case["n"] <= 150000:
        x = prepare(case, seed)["x"].double()
        k = case["min_samples"] + 1 if case["min_samples"] > 1 else 2
        core = torch.empty(len(x), dtype=torch.float64, device="cuda")
        step = max(1, int(2e9 / (8 * len(x))))
        for a in range(0, len(x), step):
            q = x[a:a + step]
            d2 = torch.zeros(len(q), len(x), dtype=torch.float64, device="cuda")
            for c in range(x.shape[1]):
                d2 += (q[:, c, None] - x[None, :, c]) ** 2
            core[a:a + step] = torch.topk(d2, k, dim=1, largest=False).values[:, -1]
        return {"core": core, "lengths": None}
    return None
