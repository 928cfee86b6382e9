"""The calls this library is measured by: one case per way it is used.

A case names an operation and a synthetic graph; ``prepare`` makes what a
program holds before the call (a resident graph, a plan, a file image), ``run``
makes the call through the package's public entry points and ``exact`` says
what it returns in plain 64-bit arithmetic.  Graphs are Graph500-style R-MATs
(a, b, c, d = .57, .19, .19, .05, symmetric, without duplicates) cut to any
vertex count, and 4-neighbour grids, as the package's generators make them;
they are made on the GPU here, so that inputs of a new seed cost little.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import graphbench_gb300 as gb

U32_UNREACHED = 0xFFFFFFFF


# ------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    return [
        # a query on a tiny graph, results in ordinary host arrays: what a call costs by itself
        {"name": "sssp_rmat_1k", "op": "sssp", "graph": "rmat", "n": 1024, "ef": 16, "w": "u32", "out": "host"},
        # an ordinary query on a skewed graph, results left on the GPU for the program's next kernel
        {"name": "sssp_rmat_200k", "op": "sssp", "graph": "rmat", "n": 200_003, "ef": 16, "w": "f32", "out": "device"},
        # the published R-MAT 22 configuration, end to end into page-locked host arrays
        {"name": "sssp_rmat_4m", "op": "sssp", "graph": "rmat", "n": 1 << 22, "ef": 16, "w": "u32", "out": "pinned"},
        # a small road-like graph: hundreds of dependent steps over little work each
        {"name": "sssp_grid_300x500", "op": "sssp", "graph": "grid", "rows": 300, "cols": 500, "w": "f32", "out": "host"},
        # the published 4096^2 grid: the largest high-diameter graph
        {"name": "sssp_grid_4096", "op": "sssp", "graph": "grid", "rows": 4096, "cols": 4096, "w": "f32", "out": "device"},
        # the reference-shaped call: a t_csr of doubles in, doubles out, the reference's delta (main/main.c:223)
        {"name": "sspath_arr_64k", "op": "sspath_arr", "graph": "rmat", "n": 1 << 16, "ef": 16, "w": "f64", "delta": 0.4},
        # many sources on one resident graph in one batched launch
        {"name": "sources_256k_64", "op": "sources", "graph": "rmat", "n": 1 << 18, "ef": 16, "w": "u32", "k": 64},
        # many small independent graphs in one batched launch
        {"name": "pack_256", "op": "pack", "graph": "rmat", "count": 256, "lo": 10, "hi": 13, "ef": 16, "w": "u32"},
        # betweenness over a sample of sources
        {"name": "bc_128k_16", "op": "bc", "graph": "rmat", "n": 131_071, "ef": 16, "w": "u32", "k": 16},
        # PageRank to convergence over in-edges
        {"name": "pagerank_1m", "op": "pagerank", "graph": "rmat", "n": 1 << 20, "ef": 16},
        # loading a binary edge list with repeated pairs into a CSR in host arrays
        {"name": "ingest_bin_256k", "op": "ingest_bin", "graph": "rmat", "n": 1 << 18, "ef": 16, "dedup": True},
        # loading a text file and answering one query on it: the reference's program from file to distances
        {"name": "text_solve_64k", "op": "text_solve", "graph": "rmat", "n": 1 << 16, "ef": 16, "delta": 0.4},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _draw_graph(rng, lo: int, hi: int) -> dict:
    """R-MAT vertex counts (or about as many grid points) between lo and hi."""
    if rng.random() < 0.35:
        side = math.isqrt(hi)
        return {"graph": "grid", "rows": _log_int(rng, 16, side), "cols": _log_int(rng, 16, side)}
    return {"graph": "rmat", "n": _log_int(rng, lo, hi), "ef": rng.choice([8, 12, 16])}


def draw(rng) -> dict:
    op = rng.choice(["sssp", "sssp", "sssp", "sspath_arr", "sources", "pack", "bc", "pagerank", "ingest_bin", "text_solve"])
    if op == "sssp":
        c = {"op": op, **_draw_graph(rng, 200, 1 << 22), "w": rng.choice(["u32", "f32", "f64"]),
             "out": rng.choice(["host", "pinned", "device"])}
        if c["graph"] == "grid":
            c["rows"], c["cols"] = _log_int(rng, 16, 4096), _log_int(rng, 16, 4096)
        if rng.random() < 0.25:      # a bucket width of the caller's own, in default widths
            c["delta_scale"] = rng.choice([0.5, 2.0, 8.0])
        return c
    if op == "sspath_arr":
        return {"op": op, "graph": "rmat", "n": _log_int(rng, 200, 1 << 17), "ef": 16, "w": rng.choice(["u32", "f64"]),
                "delta": rng.choice([0.1, 0.4])}
    if op == "sources":
        return {"op": op, **_draw_graph(rng, 1 << 10, 1 << 18), "w": rng.choice(["u32", "f32"]), "k": _log_int(rng, 2, 64)}
    if op == "pack":
        return {"op": op, "graph": "rmat", "count": _log_int(rng, 8, 256), "lo": rng.choice([8, 10]), "hi": rng.choice([11, 12, 13]),
                "ef": 16, "w": rng.choice(["u32", "f32"])}
    if op == "bc":
        return {"op": op, **_draw_graph(rng, 200, 1 << 17), "w": rng.choice(["u32", "f32", "f64"]), "k": _log_int(rng, 1, 16)}
    if op == "pagerank":
        return {"op": op, "graph": "rmat", "n": _log_int(rng, 500, 1 << 20), "ef": rng.choice([8, 16])}
    if op == "ingest_bin":
        return {"op": op, "graph": "rmat", "n": _log_int(rng, 500, 1 << 18), "ef": 16, "dedup": rng.random() < 0.5}
    return {"op": op, "graph": "rmat", "n": _log_int(rng, 500, 1 << 16), "ef": 16, "delta": rng.choice([0.1, 0.4])}


# ------------------------------------------------------------------- graphs
def _pairs(case: dict, n: int, seed: int, symmetric: bool = True):
    """(from, to) of every edge as int64 GPU tensors, in row order; not
    symmetric: 9 n different pairs and 3 n repeats of them, in random order."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    scale = max(1, (n - 1).bit_length())
    m0 = case.get("ef", 16) * n
    src = torch.zeros(m0, dtype=torch.int64, device="cuda")
    dst = torch.zeros(m0, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(m0, device="cuda", generator=gen)
        src = src * 2 + (r >= 0.76)
        dst = dst * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    perm = torch.randperm(1 << scale, device="cuda", generator=gen) % n
    src, dst = perm[src], perm[dst]
    keep = src != dst
    src, dst = src[keep], dst[keep]
    if not symmetric:
        key = torch.unique(src * n + dst)
        key = key[torch.randperm(len(key), device="cuda", generator=gen)[:9 * n]]
        key = torch.cat([key, key[torch.randint(len(key), (3 * n,), device="cuda", generator=gen)]])
        key = key[torch.randperm(len(key), device="cuda", generator=gen)]
        return key // n, key % n
    key = torch.unique(torch.cat([src * n + dst, dst * n + src]))
    return key // n, key % n


def _grid_pairs(rows: int, cols: int):
    v = torch.arange(rows * cols, device="cuda").reshape(rows, cols)
    a = torch.cat([v[:, :-1].reshape(-1), v[:-1].reshape(-1)])
    b = torch.cat([v[:, 1:].reshape(-1), v[1:].reshape(-1)])
    n = rows * cols
    key = torch.sort(torch.cat([a * n + b, b * n + a]))[0]
    return key // n, key % n


def _weights(a, b, n: int, seed: int, kind: str):
    """A weight for each undirected pair, the same in both directions: uint32
    in [1, 255], float32 in [1, 1000) on a 2^-14 lattice, or float64 in (0, 1]."""
    h = (torch.minimum(a, b) * n + torch.maximum(a, b) + ((seed * 0x632BE5AB) & 0x7FFFFFFF)) * 0x2545F4914F6CDD1D
    h = (h ^ (h >> 29)) * 0x369DEA0F31A53F85
    h = (h >> 20) & 0xFFFFFFFF
    if kind == "u32":
        return (1 + h % 255).to(torch.int32)
    if kind == "f32":
        return 1 + (h % 16367616).to(torch.float32) / 16384
    return (1 + h % 9973).to(torch.float64) / 9973


def _edges(case: dict, seed: int):
    """n, and from, to, weight of every edge in row order (GPU tensors)."""
    if case["graph"] == "grid":
        n = case["rows"] * case["cols"]
        a, b = _grid_pairs(case["rows"], case["cols"])
    else:
        n = case["n"]
        a, b = _pairs(case, n, seed)
    return n, a, b, _weights(a, b, n, seed, case.get("w", "f64"))


def _row_offsets(a, n: int):
    row = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(a, minlength=n), 0, out=row[1:])
    return row


def _host_csr(case: dict, seed: int):
    n, a, b, w = _edges(case, seed)
    row = _row_offsets(a, n).cpu().numpy().view(np.uint64)
    col = b.to(torch.int32).cpu().numpy().view(np.uint32)
    w = w.cpu().numpy()
    return row, col, w.view(np.uint32) if w.dtype == np.int32 else w


def _sources(row, k: int, seed: int):
    live = np.nonzero(np.diff(row.astype(np.int64)))[0]
    pick = np.random.default_rng(seed).choice(live, size=k, replace=len(live) < k)
    return pick.astype(np.uint32)


def _default_delta(row, w) -> float:
    return float(np.max(w)) / (len(w) / (len(row) - 1))


def _pack_cases(case: dict, seed: int):
    rng = np.random.default_rng(case["count"])   # sizes are the case's, graphs the seed's
    for i, s in enumerate(rng.uniform(case["lo"], case["hi"], size=case["count"])):
        yield {"graph": "rmat", "n": int(2 ** s), "ef": case["ef"], "w": case["w"]}, seed * 1000 + i


def _bin_image(n: int, a, b):
    """The binary edge list read_csr_bin reads (graph/csr.c:211-299), page-locked."""
    m = len(a)
    buf = gb.PinnedBuffer(32 + 16 * m, np.uint8)
    buf.array[:32].view(np.int64)[:] = (n, m, 1, n)
    pairs = torch.stack([a + 1, b + 1], 1).cpu().numpy()
    buf.array[32:].view(np.int64)[:] = pairs.reshape(-1)
    return buf


def _text_image(n: int, a, b):
    """The text scan_csr_idx and read_graph_csr read (graph/csr.c:4-202), page-locked."""
    x, y = (a + 1).cpu().numpy(), (b + 1).cpu().numpy()
    body = "".join([f"a {i} {j} 1\n" for i, j in zip(x.tolist(), y.tolist())])
    data = np.frombuffer(f"c synthetic R-MAT\np sp {n} {len(x)} 1 {n}\n{body}".encode(), dtype=np.uint8)
    buf = gb.PinnedBuffer(len(data), np.uint8)
    buf.array[:] = data
    return buf


class _OnDevice:
    """Device memory of the package's own, seen by torch."""

    def __init__(self, ptr: int, count: int, typestr: str, owner):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}
        self.owner = owner


# ----------------------------------------------------------- prepare and run
def prepare(case: dict, seed: int) -> dict:
    op = case["op"]
    s = {"op": op, "case": case}
    if op in ("sssp", "sources", "bc"):
        row, col, w = _host_csr(case, seed)
        n = len(row) - 1
        s["graph"] = gb.Graph(row, col, w)
        s["src"] = _sources(row, case.get("k", 1), seed)
        s["delta"] = case["delta_scale"] * _default_delta(row, w) if "delta_scale" in case else None
        if op == "sources":
            s["plan"] = gb.Plan(s["graph"], s["src"])
            kind = "<f4" if case["w"] == "f32" else "<i4"
            s["dist"] = torch.as_tensor(_OnDevice(s["plan"].dist.ptr.value, len(s["src"]) * n, kind, s["plan"]), device="cuda")
            s["pred"] = torch.as_tensor(_OnDevice(s["plan"].pred.ptr.value, len(s["src"]) * n, "<i4", s["plan"]), device="cuda")
        elif op == "sssp" and case["out"] == "pinned":
            s["dist"] = torch.empty(n * np.dtype(s["graph"].dist_dtype).itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(s["graph"].dist_dtype)
            s["pred"] = torch.empty(n, dtype=torch.int32, pin_memory=True).numpy()
        elif op == "sssp" and case["out"] == "device":
            kind = {"u32": torch.int32, "f32": torch.float32, "f64": torch.float64}[case["w"]]
            s["dist"] = torch.empty(n, dtype=kind, device="cuda")
            s["pred"] = torch.empty(n, dtype=torch.int32, device="cuda")
    elif op == "sspath_arr":
        row, col, w = _host_csr(case, seed)
        s["gs"] = gb.TCsr(row[1:].astype(np.int64), col.astype(np.int64), w.astype(np.float64))
        s["src"] = _sources(row, 1, seed)
    elif op == "pack":
        graphs = [gb.HostGraph(*_host_csr(c, sd)) for c, sd in _pack_cases(case, seed)]
        src = np.array([_sources(g.row, 1, seed + i)[0] for i, g in enumerate(graphs)], dtype=np.uint32)
        s["pack"] = gb.Pack(graphs)
        s["plan"] = gb.Plan(s["pack"], src)
        total = int(s["plan"].offsets[-1])
        kind = "<f4" if case["w"] == "f32" else "<i4"
        s["dist"] = torch.as_tensor(_OnDevice(s["plan"].dist.ptr.value, total, kind, s["plan"]), device="cuda")
        s["pred"] = torch.as_tensor(_OnDevice(s["plan"].pred.ptr.value, total, "<i4", s["plan"]), device="cuda")
    elif op == "pagerank":
        a, b = _pairs(case, case["n"], seed)
        image = _bin_image(case["n"], a, b)
        s["csr"] = gb.DeviceCsr.parse_bin(image.array)
    elif op == "ingest_bin":
        a, b = _pairs(case, case["n"], seed, symmetric=False)
        s["image"] = _bin_image(case["n"], a, b)
    else:
        a, b = _pairs(case, case["n"], seed)
        s["image"] = _text_image(case["n"], a, b)
        s["src"] = _sources(_row_offsets(a, case["n"]).cpu().numpy(), 1, seed)
    return s


def run(s: dict):
    op, case = s["op"], s["case"]
    if op == "sssp":
        src = int(s["src"][0])
        if case["out"] == "device":
            s["graph"].sssp_device(src, s["dist"].data_ptr(), s["pred"].data_ptr(), delta=s["delta"])
            return s["dist"], s["pred"]
        if case["out"] == "pinned":
            dist, pred, _ = s["graph"].sssp(src, delta=s["delta"], out_dist=s["dist"], out_pred=s["pred"])
        else:
            dist, pred, _ = s["graph"].sssp(src, delta=s["delta"])
        return (dist.view(np.int32) if case["w"] == "u32" else dist), pred
    if op == "sspath_arr":
        return gb.run_sspath_arr(s["gs"], int(s["src"][0]), case["delta"])
    if op in ("sources", "pack"):
        s["plan"].run()
        return s["dist"], s["pred"]
    if op == "bc":
        return s["graph"].betweenness(s["src"])[0]
    if op == "pagerank":
        rank, st = s["csr"].pagerank()
        return rank, st["iterations"]
    if op == "ingest_bin":
        with gb.DeviceCsr.parse_bin(s["image"].array, dedup=case["dedup"]) as csr:
            return csr.export()
    with gb.DeviceCsr.parse_text(s["image"].array) as csr, csr.graph(gb.W_F64) as g:
        dist, pred, _ = g.sssp(int(s["src"][0]), delta=case["delta"])
    return dist, pred


# ------------------------------------------------------------------- work
def _sizes(case: dict):
    """Vertices and, nearly, edges."""
    if case["graph"] == "grid":
        r, c = case["rows"], case["cols"]
        return r * c, 2 * (r * (c - 1) + (r - 1) * c)
    return case["n"], 1.85 * case["ef"] * case["n"]


def work(case: dict) -> dict:
    """Each edge and row offset read once, each vertex's result written once."""
    op = case["op"]
    if op == "pack":
        mean = (2 ** case["hi"] - 2 ** case["lo"]) / (math.log(2) * (case["hi"] - case["lo"])) if case["hi"] > case["lo"] else 2 ** case["lo"]
        n, m = case["count"] * mean, case["count"] * mean * 1.6 * case["ef"]
        return {"bytes": 8 * m + 12 * n, "flops": m}
    n, m = _sizes(case)
    edge = 12 if case.get("w") == "f64" else 8
    if op in ("sssp", "sspath_arr"):
        return {"bytes": edge * m + (16 if edge == 12 else 12) * n, "flops": m}
    if op == "sources":
        return {"bytes": 8 * m + 4 * n + 8 * n * case["k"], "flops": m * case["k"]}
    if op == "bc":
        return {"bytes": edge * m + 4 * n + 8 * n, "flops": 3 * m * case["k"]}
    if op == "pagerank":
        return {"bytes": 4 * m + 16 * n, "flops": 25 * m}
    if op == "ingest_bin":
        return {"bytes": 16 * 12 * n + 12 * (9 if case["dedup"] else 12) * n + 8 * n, "flops": 0}
    return {"bytes": 16 * m + 12 * n, "flops": m}


# ------------------------------------------------------------------- exact
def _distances(n: int, a, b, w, src: int):
    """Shortest distances in 64 bits by relaxing every edge until none improves."""
    d = torch.full((n,), math.inf, dtype=torch.float64, device="cuda")
    d[src] = 0
    while True:
        e = d.clone().scatter_reduce_(0, b, d[a] + w, "amin")
        if torch.equal(e, d):
            return d
        d = e


def _dependencies(n: int, a, b, d, w, src: int):
    """Brandes' dependencies of one source over its tight edges (d in the weight type's arithmetic)."""
    t = torch.isfinite(d[a]) & (d[a] + w == d[b])
    a, b = a[t], b[t]
    level = torch.zeros(n, dtype=torch.int64, device="cuda")
    while True:                      # longest path from the source, in edges
        e = level.clone().scatter_reduce_(0, b, level[a] + 1, "amax")
        if torch.equal(e, level):
            break
        level = e
    order = torch.argsort(level[a], stable=True)
    a, b = a[order], b[order]
    cut = torch.bincount(level[a]).cumsum(0).tolist() if len(a) else []
    sigma = torch.zeros(n, dtype=torch.float64, device="cuda")
    sigma[src] = 1
    lo = 0
    for hi in cut:
        sigma.index_add_(0, b[lo:hi], sigma[a[lo:hi]])
        lo = hi
    delta = torch.zeros(n, dtype=torch.float64, device="cuda")
    for k in range(len(cut) - 1, -1, -1):
        lo, hi = (cut[k - 1] if k else 0), cut[k]
        x, y = a[lo:hi], b[lo:hi]
        delta.index_add_(0, x, (1 + delta[y]) * sigma[x] / sigma[y])
    delta[src] = 0
    return delta


def _pagerank(n: int, a, b):
    """Rows a list their in-neighbours b; the reference's iteration (pagerank/pagerank_mpi.c:667-1043)."""
    recip = 1 / torch.bincount(b, minlength=n).to(torch.float64)
    weight, wb = torch.ones(n, dtype=torch.float64, device="cuda"), torch.full((n,), 0.3, dtype=torch.float64, device="cuda")
    diff = weight * recip
    while True:
        wb = wb.index_add(0, a, 0.7 * diff[b])
        diff = (wb - weight) * recip
        weight = wb
        if not bool((diff.abs() > 1e-6).any()):
            return weight


def exact(case: dict, seed: int):
    op = case["op"]
    if op in ("sssp", "sources", "pack") and case["w"] == "u32":
        return None                  # whole numbers
    if op == "pack":
        out = []
        for i, (c, sd) in enumerate(_pack_cases(case, seed)):
            n, a, b, w = _edges(c, sd)
            src = _sources(_row_offsets(a, n).cpu().numpy(), 1, seed + i)[0]
            out.append(_distances(n, a, b, w.double(), int(src)))
        return torch.cat(out), None
    if op in ("sssp", "sources"):
        if case["graph"] == "grid" and case["rows"] * case["cols"] * max(case["rows"], case["cols"]) * case.get("k", 1) > 3e9:
            return None              # thousands of steps over millions of edges
        n, a, b, w = _edges(case, seed)
        w = w.double()
        src = _sources(_row_offsets(a, n).cpu().numpy(), case.get("k", 1), seed)
        d = torch.cat([_distances(n, a, b, w, int(x)) for x in src])
        return d, None
    if op == "sspath_arr":
        n, a, b, w = _edges(case, seed)
        return _distances(n, a, b, w.double(), int(_sources(_row_offsets(a, n).cpu().numpy(), 1, seed)[0]))
    if op == "bc":
        if case["w"] == "f32" or (case["graph"] == "grid" and case["rows"] * case["cols"] * max(case["rows"], case["cols"]) * case["k"] > 3e9):
            return None              # which paths tie is decided in 32-bit sums; or too many steps
        n, a, b, w = _edges(case, seed)
        w = w.double()
        total = torch.zeros(n, dtype=torch.float64, device="cuda")
        for x in _sources(_row_offsets(a, n).cpu().numpy(), case["k"], seed):
            total += _dependencies(n, a, b, _distances(n, a, b, w, int(x)), w, int(x))
        return total
    if op == "pagerank":
        return _pagerank(case["n"], *_pairs(case, case["n"], seed)), None
    if op == "ingest_bin":
        a, b = _pairs(case, case["n"], seed, symmetric=False)
        m = len(torch.unique(a * case["n"] + b)) if case["dedup"] else len(a)
        w = torch.full((m,), 0.1, dtype=torch.float64)
        w[1::2] = 0.2
        return None, None, w
    n = case["n"]
    a, b = _pairs(case, n, seed)
    src = int(_sources(_row_offsets(a, n).cpu().numpy(), 1, seed)[0])
    return _distances(n, a, b, (b + 1).double() / n, src), None
