"""The work that users of this package have it do, as cases that can be timed.

A case names an operation of the package, a synthetic graph (family and sizes)
and the options of the call.  The families and sizes are those of the
repository's generators, tests and benchmark: R-MAT graphs with
(a, b, c) = (0.57, 0.19, 0.19) and permuted ids, road-like jittered grids,
Erdos-Renyi and Chung-Lu (exponent 2.1) graphs, seeded uniform parts.

  count        one exact count of a resident oriented graph
  per_root     the per-root counts of a resident oriented graph
  batch_parts  one batched count of a graph's resident counting-halo parts
  batch_mix    one batched count of many resident graphs of uneven sizes
  from_edges   a host edge list cleaned, oriented, downloaded and counted
  halo         halo parts extracted from a resident undirected graph, then the
               per-root counts of each
  from_csr     an oriented CSR in host memory, uploaded, validated and counted
  parts_csr    a graph's counting-halo parts in pinned host memory, uploaded,
               validated and counted
  parts_lp     a resident undirected graph partitioned by label propagation
"""
import ctypes
import math

import numpy as np
import torch

import trianglecount_gb300 as tc

A, B, C = 0.57, 0.19, 0.19
GAMMA = 2.1
P_DELETE, DIAG_RATE = 0.15, 0.05
WEDGES_MAX = 1_500_000_000  # exact() expands every wedge: more take too long


# ---- cases ---------------------------------------------------------------------
def listed():
    return [
        # one query graph of the smallest size the uneven batch holds: call and launch latency
        {"name": "small_count", "op": "count", "graph": "er", "n": 1000, "deg": 16, "tie": "reference"},
        # a road network: every oriented row fits a lane's registers
        {"name": "road_count", "op": "count", "graph": "road", "side": 1448, "height": 1448, "tie": "reference"},
        # a small social graph, counted again and again: short kernels
        {"name": "rmat16_count", "op": "count", "graph": "rmat", "scale": 16, "ef": 16, "tie": "reference"},
        # the ordinary large social graph of TC_128
        {"name": "rmat21_count", "op": "count", "graph": "rmat", "scale": 21, "ef": 16, "tie": "reference"},
        # g_sum of every vertex, as for clustering coefficients
        {"name": "chung_lu_per_root", "op": "per_root", "graph": "chung_lu", "n": 1_000_000, "deg": 16, "tie": "id_asc"},
        # the benchmark's headline: eight halo parts of the largest graph in one launch
        {"name": "rmat23_parts", "op": "batch_parts", "graph": "rmat", "scale": 23, "ef": 16, "k": 8, "tie": "reference"},
        # many query graphs of all sizes and families in one launch
        {"name": "uneven_batch", "op": "batch_mix", "graphs": 64, "tie": "reference"},
        # tc_preprocess: an edge list with both directions, repeats and self-loops becomes an oriented CSR
        {"name": "edges_to_csr", "op": "from_edges", "graph": "rmat", "scale": 18, "ef": 16, "tie": "reference"},
        # round_clean_sg and wo_sort_tc_256 without the files between them
        {"name": "halo_parts", "op": "halo", "graph": "rmat", "scale": 20, "ef": 16, "k": 8, "mode": "reference",
         "tie": "reference"},
        # a u64 part file of wo_sort_tc_256 as it was read, counted once
        {"name": "csr_u64_count", "op": "from_csr", "graph": "rmat", "scale": 19, "ef": 16, "dtype": "uint64",
         "tie": "reference"},
        # the partitioned count end to end from host memory
        {"name": "parts_from_host", "op": "parts_csr", "graph": "rmat", "scale": 21, "ef": 16, "k": 8, "tie": "reference"},
        # the stand-in for METIS on a social graph
        {"name": "label_parts", "op": "parts_lp", "graph": "chung_lu", "n": 500_000, "deg": 16, "k": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, families, edges_max):
    """A graph of one of the families with at most edges_max edges."""
    f = rng.choice(families)
    if f == "rmat":
        ef = rng.randint(8, 24)
        return {"graph": f, "scale": rng.randint(10, int(math.log2(edges_max / ef))), "ef": ef}
    if f == "road":
        side = _log_int(rng, 33, math.sqrt(edges_max / 1.75))
        return {"graph": f, "side": side, "height": max(2, int(side * rng.uniform(0.5, 1.0)))}
    deg = rng.randint(8, 64)
    lo = 1000 if f == "er" else 10_000
    return {"graph": f, "n": _log_int(rng, lo, min(4_000_000, 2 * edges_max / deg)), "deg": deg}


def draw(rng):
    every = ["er", "road", "rmat", "chung_lu"]
    op = rng.choice(["count", "count", "count", "per_root", "batch_parts", "batch_mix", "from_edges", "halo", "from_csr",
                     "parts_csr", "parts_lp"])
    tie = rng.choice(["reference", "id_asc"])
    if op in ("count", "per_root"):
        return {"op": op, **_draw_graph(rng, every, 40_000_000), "tie": tie}
    if op in ("batch_parts", "parts_csr"):
        return {"op": op, **_draw_graph(rng, ["rmat", "rmat", "chung_lu"], 34_000_000), "k": rng.randint(2, 8), "tie": tie}
    if op == "batch_mix":
        return {"op": op, "graphs": rng.randint(2, 64), "tie": tie}
    if op == "from_edges":
        return {"op": op, **_draw_graph(rng, every, 8_000_000), "tie": tie}
    if op == "halo":
        return {"op": op, **_draw_graph(rng, every, 17_000_000), "k": rng.randint(2, 12),
                "mode": rng.choice(["reference", "count"]), "tie": tie}
    if op == "from_csr":
        return {"op": op, **_draw_graph(rng, every, 17_000_000), "dtype": rng.choice(["int32", "uint64"]), "tie": tie}
    return {"op": op, **_draw_graph(rng, every, 8_000_000), "k": rng.randint(2, 16)}


# ---- inputs ---------------------------------------------------------------------
def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)


def _rmat(scale, ef, g):
    m = ef << scale
    u = torch.zeros(m, dtype=torch.int64, device="cuda")
    v = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, generator=g, device="cuda")
        ub = r >= A + B
        vb = ((r >= A) & ~ub) | (r >= A + B + C)
        u = 2 * u + ub
        v = 2 * v + vb
    perm = torch.randperm(1 << scale, generator=g, device="cuda")
    return perm[u], perm[v]


def _er(n, deg, g):
    m = max(1, n * deg // 2)
    return (torch.randint(n, (m,), generator=g, device="cuda"), torch.randint(n, (m,), generator=g, device="cuda"))


def _chung_lu(n, deg, g):
    m = max(1, n * deg // 2)
    w = torch.arange(1, n + 1, dtype=torch.float64, device="cuda") ** (-1.0 / (GAMMA - 1.0))
    w = torch.clamp(w * (n * deg / w.sum()), max=math.sqrt(2.0 * m))
    cum = torch.cumsum(w, 0)
    ends = [torch.searchsorted(cum, torch.rand(m, generator=g, device="cuda", dtype=torch.float64) * cum[-1]).clamp(max=n - 1)
            for _ in range(2)]
    perm = torch.randperm(n, generator=g, device="cuda")
    return perm[ends[0]], perm[ends[1]]


def _road(side, height, g):
    v = torch.arange(side * height, device="cuda").reshape(height, side)

    def kept(t, p):
        t = t.reshape(-1)
        return t[torch.rand(t.numel(), generator=g, device="cuda") < p]

    right = kept(v[:, :-1], 1 - P_DELETE)
    down = kept(v[:-1, :], 1 - P_DELETE)
    diag = kept(v[:-1, :-1], DIAG_RATE)
    return torch.cat((right, down, diag)), torch.cat((right + 1, down + side, diag + side + 1))


def _edges(case, seed):
    """The graph's edge list on the GPU, int64."""
    g = _rng(seed)
    f = case["graph"]
    if f == "rmat":
        return _rmat(case["scale"], case["ef"], g)
    if f == "er":
        return _er(case["n"], case["deg"], g)
    if f == "chung_lu":
        return _chung_lu(case["n"], case["deg"], g)
    return _road(case["side"], case["height"], g)


def _host_edges(case, seed):
    return tuple(t.cpu().numpy() for t in _edges(case, seed))


def _mix(case, seed):
    """The uneven batch: a third each of Erdos-Renyi, Chung-Lu and R-MAT graphs, sizes log-uniform."""
    r = np.random.default_rng(seed)
    out = []
    for i in range(case["graphs"]):
        deg = int(r.integers(8, 65))
        if i % 3 == 0:
            c = {"graph": "er", "n": int(round(math.exp(r.uniform(math.log(1e3), math.log(1e5))))), "deg": deg}
        elif i % 3 == 1:
            c = {"graph": "chung_lu", "n": int(round(math.exp(r.uniform(math.log(1e4), math.log(1e6))))), "deg": deg}
        else:
            c = {"graph": "rmat", "scale": int(r.integers(10, 19)), "ef": 16}
        out.append((c, int(r.integers(1 << 40))))
    return out


def _parts_of(n, k, seed):
    return np.random.default_rng(seed).integers(0, k, n, dtype=np.int32)


def _pinned(a):
    t = torch.empty(len(a), dtype=torch.int32, pin_memory=True).numpy()
    t[:] = a
    return t


def _address(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _check(status):
    if status:
        raise RuntimeError(tc.lib().tc_last_error().decode())


_CTX = None


def _ctx():
    """A program's one context."""
    global _CTX
    if _CTX is None:
        _CTX = tc.Context(0)
    return _CTX


def prepare(case, seed):
    ctx, op = _ctx(), case["op"]
    s = {"op": op, "ctx": ctx, "tie": case.get("tie")}
    if op == "batch_mix":
        graphs = [ctx.graph_from_edges(*_host_edges(c, q), tie=case["tie"]) for c, q in _mix(case, seed)]
        s["batch"] = ctx.batch(graphs)
        return s
    src, dst = _host_edges(case, seed)
    ids = _size(case)[0]  # result buffers are sized for the id space, as a caller of the C ABI does before the clean-up
    if op == "from_edges":  # as collected: some edges both ways, some twice, some self-loops
        n = len(src) // 16
        s["rp"], s["col"] = np.zeros(ids + 1, np.int32), np.zeros(len(src), np.int32)
        s["src"] = np.concatenate((src, dst[:n], src[n:2 * n], src[:n // 8]))
        s["dst"] = np.concatenate((dst, src[:n], dst[n:2 * n], src[:n // 8]))
        return s
    if op in ("count", "per_root"):
        s["graph"] = ctx.graph_from_edges(src, dst, tie=case["tie"])
        s["per_root"] = np.zeros(ids, np.uint64)
        return s
    if op == "from_csr":
        rp, col = ctx.graph_from_edges(src, dst, tie=case["tie"]).download()
        s["rp"], s["col"] = rp.astype(case["dtype"]), col.astype(case["dtype"])
        return s
    ug = ctx.ugraph_from_edges(src, dst)
    if op == "parts_lp":
        s.update(ug=ug, k=case["k"], seed=seed, part=np.zeros(ids, np.int32))
        return s
    part = _parts_of(ug.info()[0], case["k"], seed)
    if op == "halo":
        s.update(ug=ug, part=part, k=case["k"], mode=case["mode"], per_root=np.zeros(ids, np.uint64))
        return s
    parts = ctx.halo_extract(ug, part, case["k"], tie=case["tie"], mode="count")
    if op == "batch_parts":
        s["batch"] = ctx.batch(parts)
        return s
    s["parts"] = [(*(_pinned(a) for a in p.download()), p.n_roots) for p in parts]
    return s


def _per_root(ctx, graph, out):
    total = ctypes.c_uint64()
    _check(tc.lib().tc_count_per_root(ctx.handle, graph.handle, _address(out), ctypes.byref(total)))


def run(s):
    ctx, op = s["ctx"], s["op"]
    if op == "count":
        return ctx.count(s["graph"])
    if op == "per_root":
        _per_root(ctx, s["graph"], s["per_root"])
        return s["per_root"]
    if op in ("batch_parts", "batch_mix"):
        return s["batch"].run()
    if op == "from_edges":
        g = ctx.graph_from_edges(s["src"], s["dst"], tie=s["tie"])
        _check(tc.lib().tc_graph_download_i32(ctx.handle, g.handle, _address(s["rp"]), _address(s["col"])))
        return s["rp"], s["col"], ctx.count(g)
    if op == "halo":  # the parts' roots one after the other
        at = 0
        for p in ctx.halo_extract(s["ug"], s["part"], s["k"], tie=s["tie"], mode=s["mode"]):
            roots = p.n_roots
            _per_root(ctx, p, s["per_root"][at:at + roots])
            at += roots
        return s["per_root"]
    if op == "from_csr":
        if s["rp"].dtype == np.uint64:
            return ctx.count(ctx.upload(s["rp"], s["col"]))
        return ctx.count_csr(s["rp"], s["col"])
    if op == "parts_csr":
        return ctx.count_parts_csr(s["parts"])
    _check(tc.lib().tc_gen_parts_lp(ctx.handle, s["ug"].handle, s["k"], s["seed"], 20, _address(s["part"])))
    return s["part"]


# ---- what a pass cannot do without ------------------------------------------------
def _size(c):
    """(vertices, edges) of a graph before the clean-up."""
    f = c["graph"]
    if f == "rmat":
        return 1 << c["scale"], c["ef"] << c["scale"]
    if f == "road":
        n = c["side"] * c["height"]
        return n, int(n * (2 * (1 - P_DELETE) + DIAG_RATE))
    return c["n"], max(1, c["n"] * c["deg"] // 2)


def work(case):
    """Bytes of the inputs and outputs (sizes before the clean-up); the arithmetic is whole-number compares."""
    op = case["op"]
    if op == "batch_mix":  # the means of the three families' sizes
        v, e = case["graphs"] * 100_000, case["graphs"] * 1_800_000
        return {"bytes": 4 * v + 4 * e + 8 * case["graphs"], "flops": 0}
    v, e = _size(case)
    if op == "count":
        return {"bytes": 4 * v + 4 * e + 8, "flops": 0}
    if op == "per_root":
        return {"bytes": 12 * v + 4 * e, "flops": 0}
    if op == "from_edges":
        return {"bytes": 18 * e + 4 * v + 4 * e + 8, "flops": 0}
    if op == "halo":  # the undirected CSR and the part map in, the per-root counts out
        return {"bytes": 4 * v + 8 * e + 4 * v + 8 * v, "flops": 0}
    if op == "from_csr":
        return {"bytes": (8 if case["dtype"] == "uint64" else 4) * (v + e) + 8, "flops": 0}
    if op == "parts_lp":
        return {"bytes": 4 * v + 8 * e + 4 * v, "flops": 0}
    held = 1 + 0.75 * (case["k"] - 1)  # edges that the parts of a skewed graph hold, over the graph's
    return {"bytes": held * (4 * v + 4 * e) + 8 * case["k"], "flops": 0}


# ---- the same results from plain torch -----------------------------------------------
def _clean(src, dst):
    """Simple undirected edges (both directions, sorted) over the non-isolated vertices, relabelled in order."""
    keep = src != dst
    src, dst = src[keep], dst[keep]
    n = int(max(src.max(), dst.max())) + 1 if src.numel() else 1
    key = torch.unique(torch.cat((src * n + dst, dst * n + src)))
    u, v = key // n, key % n
    ids = torch.unique(u)
    return torch.searchsorted(ids, u), torch.searchsorted(ids, v), ids.numel()


def _orient(u, v, n, tie):
    deg = torch.bincount(u, minlength=n)
    du, dv = deg[u], deg[v]
    low = v < u if tie == "reference" else u < v
    keep = (du < dv) | ((du == dv) & low)
    return u[keep], v[keep]


def _count(u, v, n):
    """Per-root counts of an oriented edge list sorted by (u, v), every wedge looked up; None when there are too many."""
    d = torch.bincount(u, minlength=n)
    rp = torch.cat((torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(d, 0)))
    key = u * n + v
    wedges = torch.cumsum(d[v], 0)
    if not u.numel():
        return torch.zeros(n, dtype=torch.int64, device="cuda")
    if int(wedges[-1]) > WEDGES_MAX:
        return None
    out = torch.zeros(n, dtype=torch.int64, device="cuda")
    step = 1 << 26
    for a in range(0, int(wedges[-1]), step):
        t = torch.arange(a, min(a + step, int(wedges[-1])), device="cuda")
        e = torch.searchsorted(wedges, t, right=True)
        w = v[rp[v[e]] + t - (wedges[e] - d[v[e]])]
        want = u[e] * n + w
        at = torch.searchsorted(key, want).clamp(max=key.numel() - 1)
        out += torch.bincount(u[e][key[at] == want], minlength=n)
    return out


def exact(case, seed):
    op = case["op"]
    if op == "batch_mix":
        if case["graphs"] > 8:
            return None
        each = []
        for c, q in _mix(case, seed):
            u, v, n = _clean(*_edges(c, q))
            r = _count(*_orient(u, v, n, case["tie"]), n)
            if r is None:
                return None
            each.append(int(r.sum()))
        return np.array(each, np.uint64)
    if op == "parts_lp" or _size(case)[1] > 20_000_000:
        return None
    u, v, n = _clean(*_edges(case, seed))
    ou, ov = _orient(u, v, n, case["tie"])
    r = _count(ou, ov, n)
    if r is None:
        return None
    host = r.cpu().numpy().astype(np.uint64)
    ids = _size(case)[0]
    if op in ("count", "from_csr"):
        return int(host.sum())
    if op == "per_root":
        return np.pad(host, (0, ids - n))
    if op == "from_edges":
        rp = np.concatenate(([0], np.cumsum(np.bincount(ou.cpu().numpy(), minlength=n)))).astype(np.int32)
        col = ov.cpu().numpy().astype(np.int32)
        return np.pad(rp, (0, ids - n)), np.pad(col, (0, len(_edges(case, seed)[0]) - len(col))), int(host.sum())
    part = _parts_of(n, case["k"], seed)
    if op == "halo":
        return np.pad(np.concatenate([host[part == p] for p in range(case["k"])]), (0, ids - n))
    return np.array([host[part == p].sum() for p in range(case["k"])], np.uint64)
