"""Performance cases: the work a program has this package do, through its
public entry points, over the range of graphs the package is used on.

A case is a dict of plain values:
  kind   "exact"   gpu_exact_triangle_count on a CSR in device memory
         "hybrid"  gpu_hybrid_triangle_count on a CSR and its dense sketches
         "sketch"  zeroed dense sketches of a CSR and build_sketches_kernel
         "csr"     csr_from_edge_list on raw endpoint arrays
         "batch"   GraphBatch.hybrid_counts over many graphs
  graph  "rmat" (scale, ef), "er" (n, raw), "lattice" (rows, cols)
  p, theta, gamma   HLL precision and the sketch / routing thresholds
  graphs the batch size (lognormal sizes, half Erdos-Renyi, half Chung-Lu)
"""
from __future__ import annotations

import random

import torch

from triangle_counting_hll_b200 import batch, core
from triangle_counting_hll_b200.gpu_graph import csr_from_edge_list
from triangle_counting_hll_b200.gpu_hll import alloc_sketch_arrays_device, build_sketches_kernel
from triangle_counting_hll_b200.gpu_hybrid import gpu_exact_triangle_count, gpu_hybrid_triangle_count

MAX_RAW = 1 << 26          # raw edges of the largest graph (R-MAT scale 22, edge factor 16)
MAX_SKETCH_BYTES = 10 << 30


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest graph a query asks for: launches and host time
        {"name": "exact_rmat_12", "kind": "exact", "graph": "rmat", "scale": 12, "ef": 16},
        # road-like network: a million vertices, every list at most six long
        {"name": "exact_lattice_1000", "kind": "exact", "graph": "lattice", "rows": 1000, "cols": 1000},
        # a middling query of a serving mix, odd edge factor
        {"name": "exact_rmat_17", "kind": "exact", "graph": "rmat", "scale": 17, "ef": 21},
        # the headline graph: 64 M oriented edges, hubs of 1e5 neighbours
        {"name": "exact_rmat_22", "kind": "exact", "graph": "rmat", "scale": 22, "ef": 16},
        # small sparse graph with a hybrid query that finds no long list
        {"name": "hybrid_er_20k", "kind": "hybrid", "graph": "er", "n": 20000, "raw": 100000, "p": 10,
         "theta": 16, "gamma": 16},
        # the hybrid query of a serving mix (p = 12, threshold 128)
        {"name": "hybrid_rmat_18_p12", "kind": "hybrid", "graph": "rmat", "scale": 18, "ef": 24, "p": 12,
         "theta": 128, "gamma": 128},
        # the precision that keeps the estimate within 2% on skewed graphs
        {"name": "hybrid_rmat_19_p14", "kind": "hybrid", "graph": "rmat", "scale": 19, "ef": 16, "p": 14,
         "theta": 256, "gamma": 256},
        # the headline graph, estimated
        {"name": "hybrid_rmat_22_p12", "kind": "hybrid", "graph": "rmat", "scale": 22, "ef": 16, "p": 12,
         "theta": 256, "gamma": 256},
        # the sketches of the headline graph, in the zeroed arrays a program allocates for them
        {"name": "sketch_rmat_22_p10", "kind": "sketch", "graph": "rmat", "scale": 22, "ef": 16, "p": 10,
         "theta": 256},
        # loading: a small edge list and the headline one
        {"name": "csr_rmat_13", "kind": "csr", "graph": "rmat", "scale": 13, "ef": 11},
        {"name": "csr_rmat_22", "kind": "csr", "graph": "rmat", "scale": 22, "ef": 16},
        # 2,048 graphs in one call: sketches, exact and HLL edges of each
        {"name": "batch_2048", "kind": "batch", "graphs": 2048, "p": 10, "theta": 64, "gamma": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_rmat(rng, max_scale):
    scale = rng.randint(12, max_scale)
    ef = rng.randint(8, min(32, (MAX_RAW >> scale) - 1))
    return {"graph": "rmat", "scale": scale, "ef": ef}


def draw(rng):
    kind = rng.choice(["exact", "exact", "hybrid", "hybrid", "sketch", "csr", "csr", "batch"])
    c = {"kind": kind}
    if kind == "exact":
        if rng.random() < 0.3:
            c.update(graph="lattice", rows=_log_int(rng, 60, 1400), cols=_log_int(rng, 60, 1400))
        else:
            c.update(_draw_rmat(rng, 22))
    elif kind == "hybrid":
        if rng.random() < 0.25:
            n = _log_int(rng, 3000, 300000)
            c.update(graph="er", n=n, raw=int(n * rng.uniform(4.0, 16.0)), p=10, theta=16, gamma=16)
        else:
            p = rng.choice([8, 10, 12, 14])
            t = rng.choice([64, 128, 256])
            c.update(_draw_rmat(rng, 21))
            while p > 8 and (1 << (c["scale"] + p)) > MAX_SKETCH_BYTES:
                p -= 2
            c.update(p=p, theta=t, gamma=t)
    elif kind == "sketch":
        c.update(_draw_rmat(rng, 21))
        p = rng.choice([8, 10, 12, 14])
        while p > 8 and (1 << (c["scale"] + p)) > MAX_SKETCH_BYTES // 4:
            p -= 2
        c.update(p=p, theta=rng.choice([64, 128, 256]))
    elif kind == "csr":
        if rng.random() < 0.25:
            n = _log_int(rng, 3000, 3000000)
            c.update(graph="er", n=n, raw=int(n * rng.uniform(2.0, 10.0)))
        else:
            c.update(_draw_rmat(rng, 22))
    else:
        c.update(graphs=_log_int(rng, 48, 1500), p=10, theta=64, gamma=64)
    return c


# ------------------------------------------------------------------ inputs
def _edges(case, seed):
    if case["graph"] == "rmat":
        return core.gen_rmat(case["scale"], case["ef"], 0.57, 0.19, 0.19, seed=seed)
    if case["graph"] == "er":
        return core.gen_er(case["n"], case["raw"], seed=seed)
    return core.gen_lattice(case["rows"], case["cols"], seed=seed)


def _relabelled(case, seed):
    """The edges of one graph under other ids (every id XOR one mask: n and m
    stay, so outputs of a size that depends on the graph keep it, and the
    ids keep their locality) and from another starting point of the list."""
    u, v = _edges(case, 1)
    rng = random.Random(seed)
    mask = rng.randrange(1, 1 << max(1, int(torch.maximum(u.max(), v.max())).bit_length()))
    at = rng.randrange(u.numel())
    return torch.roll(u ^ mask, at), torch.roll(v ^ mask, at)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "csr":
        u, v = _relabelled(case, seed)
        return {"case": case, "u": u, "v": v}
    if kind == "batch":
        specs = batch.c4_specs(case["graphs"], seed_base=seed % 1000003)
        lists = []
        for s in specs:
            u, v = batch.generate(s)
            lists.append((u, v, s.n))
        return {"case": case, "batch": batch.GraphBatch.from_edge_lists(lists)}
    g = core.csr_from_edges(*(_relabelled(case, seed) if kind == "sketch" else _edges(case, seed)))
    state = {"case": case, "csr": g}
    if kind == "hybrid":
        regs, has = alloc_sketch_arrays_device(g.n_nodes, case["p"])
        build_sketches_kernel[(g.n_nodes + 255) // 256, 256](g.row_ptr, g.col_idx, g.n_nodes, case["theta"],
                                                             case["p"], regs, has)
        state.update(regs=regs, has=has)
    return state


# ---------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "csr":
        return csr_from_edge_list(state["u"], state["v"])
    if kind == "batch":
        totals, stats = state["batch"].hybrid_counts(case["theta"], case["gamma"], case["p"])
        return {"total": totals, **stats}
    g = state["csr"]
    if kind == "exact":
        count, _ = gpu_exact_triangle_count(g.row_ptr, g.col_idx, g.edge_u, g.edge_v)
        return {"count": count}
    if kind == "hybrid":
        total, _, stats = gpu_hybrid_triangle_count(g.row_ptr, g.col_idx, g.edge_u, g.edge_v, g.degrees,
                                                    state["regs"], state["has"], case["gamma"], case["p"])
        return {"total": total, "n_approx": stats["n_approx"], "n_exact": stats["n_exact"],
                "n_clamped": stats["n_clamped"]}
    regs, has = alloc_sketch_arrays_device(g.n_nodes, case["p"])
    build_sketches_kernel[(g.n_nodes + 255) // 256, 256](g.row_ptr, g.col_idx, g.n_nodes, case["theta"], case["p"],
                                                         regs, has)
    return {"regs": regs, "has": has}


# -------------------------------------------------------------------- work
def _size(case):
    """(vertices, oriented edges), about."""
    if case["kind"] == "batch":
        raw = 49500.0 * case["graphs"]
        return raw / 6.0, 0.95 * raw
    if case["graph"] == "lattice":
        n = case["rows"] * case["cols"]
        return float(n), 2.2 * n
    if case["graph"] == "er":
        return float(case["n"]), float(case["raw"])
    raw = case["ef"] << case["scale"]
    return 0.6 * (1 << case["scale"]), (0.75 + 0.02 * (case["scale"] - 12)) * raw


def work(case):
    n, m = _size(case)
    kind = case["kind"]
    if kind == "csr":  # raw endpoints in; row_ptr, degrees, ids, col_idx, edge_u, edge_v out
        raw = case["raw"] if case["graph"] == "er" else (case["ef"] << case["scale"])
        return {"bytes": 8.0 * raw + 12.0 * n + 12.0 * m, "flops": 0.0}
    if kind == "sketch":  # row_ptr and the lists in, every register and flag out
        return {"bytes": 4.0 * n + 4.0 * m + n * ((1 << case["p"]) + 1), "flops": 0.0}
    b = 4.0 * n + 12.0 * m
    if kind == "hybrid":  # + degrees, flags and the rows of the sketched vertices
        rows = 0.0 if case["graph"] == "er" else 0.005 * n + 0.1 * m / case["theta"]
        b += 5.0 * n + rows * (1 << case["p"])
    return {"bytes": b, "flops": 0.0}


# ------------------------------------------------- the results, in 64 bits
def _support(row_ptr, col, eu, ev, n):
    """|N+(u) cap N+(v)| of every edge: each member w of the shorter list is
    looked up as the edge (other endpoint, w) among the sorted edge keys."""
    deg = row_ptr[1:] - row_ptr[:-1]
    keys = torch.repeat_interleave(torch.arange(n, device=col.device), deg) * n + col
    swap = deg[eu] < deg[ev]
    x, y = torch.where(swap, ev, eu), torch.where(swap, eu, ev)
    cum = torch.cumsum(deg[y], 0)
    out = torch.zeros(eu.numel(), dtype=torch.int64, device=col.device)
    lo = 0
    while lo < eu.numel():
        base = int(cum[lo - 1]) if lo else 0
        hi = max(lo + 1, int(torch.searchsorted(cum, base + (1 << 27), right=True)))
        d = deg[y[lo:hi]]
        e = torch.repeat_interleave(torch.arange(hi - lo, device=col.device), d)
        k = torch.arange(e.numel(), device=col.device) - (torch.cumsum(d, 0) - d)[e]
        q = x[lo:hi][e] * n + col[row_ptr[y[lo:hi]][e] + k]
        at = torch.searchsorted(keys, q).clamp_(max=max(keys.numel() - 1, 0))
        out[lo:hi].index_add_(0, e, (keys[at] == q).to(torch.int64))
        lo = hi
    return out


def _hash(x):
    def shr(v, s):
        return (v >> s) & ((1 << (64 - s)) - 1)
    x = (x ^ shr(x, 30)) * (0xBF58476D1CE4E5B9 - (1 << 64))
    x = (x ^ shr(x, 27)) * (0x94D049BB133111EB - (1 << 64))
    return x ^ shr(x, 31)


def _registers(row_ptr, ids, sketched, p):
    """One register row per sketched vertex, from the ids in its list."""
    m, rem = 1 << p, 64 - p
    rank = torch.full((row_ptr.numel() - 1,), -1, dtype=torch.int64, device=ids.device)
    rank[sketched] = torch.arange(sketched.numel(), device=ids.device)
    own = torch.repeat_interleave(rank, row_ptr[1:] - row_ptr[:-1])
    h = _hash(ids[own >= 0])
    j = (h >> rem) & (m - 1)
    w = h & ((1 << rem) - 1)
    bits = torch.zeros_like(w)
    for s in (32, 16, 8, 4, 2, 1):
        big = (w >> s) > 0
        bits += torch.where(big, s, 0)
        w = torch.where(big, w >> s, w)
    bits += w
    rows = torch.zeros(sketched.numel() * m, dtype=torch.int64, device=ids.device)
    rows.scatter_reduce_(0, own[own >= 0] * m + j, rem - bits + 1, "amax")
    return rows.view(-1, m), rank


def _estimate(rows, a, b, p):
    """Union estimates of rows[a] and rows[b] in double precision."""
    m = 1 << p
    alpha = {16: 0.673, 32: 0.697, 64: 0.709}.get(m, 0.7213 / (1.0 + 1.079 / m))
    inv = torch.pow(torch.tensor(2.0, dtype=torch.float64, device=rows.device),
                    -torch.arange(66, device=rows.device, dtype=torch.float64))
    out = torch.empty(a.numel(), dtype=torch.float64, device=rows.device)
    step = max(1, (1 << 27) >> p)
    for lo in range(0, a.numel(), step):
        r = torch.maximum(rows[a[lo:lo + step]], rows[b[lo:lo + step]])
        z = inv[r.to(torch.int64)].sum(1)
        v = (r == 0).sum(1).to(torch.float64)
        e = alpha * m * m / z
        out[lo:lo + step] = torch.where((e <= 2.5 * m) & (v > 0), m * torch.log(m / v.clamp(min=1.0)), e)
    return out


def _hybrid(row_ptr, col, eu, ev, deg, sketched, rows, rank, gamma, p, graph, n_graphs):
    n = row_ptr.numel() - 1
    proxy = torch.minimum(deg[eu], deg[ev])
    hll = (proxy >= gamma) & sketched[eu] & sketched[ev]
    wants = proxy >= gamma
    ex = ~hll
    zero = torch.zeros(n_graphs, dtype=torch.int64, device=col.device)
    exact = zero.clone().index_add_(0, graph[ex], _support(row_ptr, col, eu[ex], ev[ex], n))
    a, b = eu[hll], ev[hll]
    s = (deg[a] + deg[b]).to(torch.float64) - _estimate(rows, rank[a], rank[b], p)
    top = proxy[hll].to(torch.float64)
    part = torch.zeros(n_graphs, dtype=torch.float64, device=col.device)
    part.index_add_(0, graph[hll], torch.minimum(s, top).clamp(min=0.0))

    def per_graph(mask, idx):
        return zero.clone().index_add_(0, idx, mask.to(torch.int64))
    return {"total": exact.to(torch.float64) + part, "n_approx": per_graph(hll, graph),
            "n_exact": per_graph(ex, graph), "n_fallback": per_graph(wants & ~hll, graph),
            "n_clamped": per_graph((s < 0) | (s > top), graph[hll])}


def exact(case, seed):
    """Hybrid totals in double precision; the other kinds return integers."""
    if case["kind"] not in ("hybrid", "batch") or _size(case)[1] > 1.2e8:
        return None
    if case["kind"] == "hybrid" and case["graph"] == "rmat" and case["ef"] << case["scale"] > 1 << 24:
        return None  # minutes of work for plain tensor operations
    state = prepare(case, seed)
    p = case["p"]
    if case["kind"] == "batch":
        g, vb = state["batch"].csr, state["batch"].vbase.to(torch.int64)
        row_ptr, col = g.row_ptr.to(torch.int64), g.col_idx.to(torch.int64)
        deg = row_ptr[1:] - row_ptr[:-1]
        owner = torch.repeat_interleave(torch.arange(vb.numel() - 1, device=col.device), vb[1:] - vb[:-1])
        eu = torch.repeat_interleave(torch.arange(g.n_nodes, device=col.device), deg)
        sketched = deg >= case["theta"]
        rows, rank = _registers(row_ptr, col - vb[owner[col]], sketched.nonzero().view(-1), p)
        return _hybrid(row_ptr, col, eu, col, deg, sketched, rows, rank, case["gamma"], p, owner[eu], vb.numel() - 1)
    g = state["csr"]
    row_ptr, col = g.row_ptr.to(torch.int64), g.col_idx.to(torch.int64)
    deg = row_ptr[1:] - row_ptr[:-1]
    sketched = deg >= case["theta"]
    ids = torch.arange(g.n_nodes, device=col.device)
    rows, rank = state["regs"].view(g.n_nodes, 1 << p), ids
    eu = torch.repeat_interleave(ids, deg)
    r = _hybrid(row_ptr, col, eu, col, deg, sketched, rows, rank, case["gamma"], p, torch.zeros_like(eu), 1)
    return {"total": float(r["total"][0]), "n_approx": int(r["n_approx"][0]), "n_exact": int(r["n_exact"][0]),
            "n_clamped": int(r["n_clamped"][0])}
