"""Timed cases of the engine's public entry points.

Every case is one call (or one loop of calls) that a program written against
``fastapsp_gb300`` makes: all-pairs solves of the three graph families with
the rows kept on the device, the part-by-part loop of graphs too large for one
result, the drop-in class with host results, the batched Floyd-Warshall
forward and its adjoint, the (min,+) product, multi-source shortest paths, and
the consumers of solved rows (queries and the weight gradient).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import fastapsp_gb300 as fap
from fastapsp_gb300 import graphs

INF_I32 = 1 << 30
INF_F32 = 1e8


def listed():
    return [
        # The smallest solve a program makes (one call per small map or test graph): launches and latency.
        {"name": "solve_grid_small", "kind": "solve", "graph": "grid", "rows": 24, "cols": 24, "parts": 4},
        # Hop counts of an undirected grid, all pairs, rows on the device.
        {"name": "solve_grid", "kind": "solve", "graph": "grid", "rows": 128, "cols": 128, "parts": 16},
        # A directed nearest-neighbour graph with integer weights: most pairs unreachable.
        {"name": "solve_geometric", "kind": "solve", "graph": "geometric", "n": 65536, "parts": 64},
        # A road network with real weights and exactly summed boundary rows, odd row length; the largest case.
        {"name": "solve_road", "kind": "solve", "graph": "road", "n": 57301, "parts": 64},
        # Graphs past the split limit of the drop-in class: one part at a time, the reference's FP32 arithmetic.
        {"name": "parts_road", "kind": "parts", "n": 24575, "parts": 27},
        # The drop-in class: fapGraph.solve() into host rows.
        {"name": "dropin_road", "kind": "dropin", "n": 4801, "parts": 6},
        # Batched Floyd-Warshall of dense integer instances of very different sizes (forward only).
        {"name": "floyd_dense", "kind": "floyd", "count": 512, "nmin": 32, "nmax": 2048},
        # Forward and backward over a batch of sparse real-weight digraphs: Floyd-Warshall, then the adjoint.
        {"name": "floyd_adjoint", "kind": "adjoint", "count": 256, "nmin": 256, "nmax": 1024, "pairs": 10000},
        # The product that extends a part's inner rows: few steps, many columns, rows of odd length.
        {"name": "minplus_wide_f32", "kind": "minplus", "dtype": "f32", "m": 877, "n": 114599, "k": 19},
        # A square integer distance product with predecessors, steps past the packed range.
        {"name": "minplus_deep_i32", "kind": "minplus", "dtype": "i32", "m": 1000, "n": 4000, "k": 500},
        # Shortest paths from a few dozen sources of a large road network, FP32.
        {"name": "sssp_road", "kind": "sssp", "n": 114599, "sources": 64},
        # Consumers of solved rows: point-to-point paths and the gradient on the edge weights.
        {"name": "paths_road", "kind": "paths", "n": 4096, "parts": 4, "pairs": 10000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["solve_grid", "solve_geometric", "solve_road", "parts", "dropin", "floyd", "adjoint",
                       "minplus_f32", "minplus_i32", "sssp", "paths"])
    if kind == "solve_grid":
        rows = _log_int(rng, 20, 160)
        cols = max(20, min(200, int(rows * rng.uniform(0.6, 1.6))))
        return {"kind": "solve", "graph": "grid", "rows": rows, "cols": cols,
                "parts": max(2, rows * cols // rng.randint(700, 1100))}
    if kind in ("solve_geometric", "solve_road"):
        n = _log_int(rng, 1500, 55000)
        return {"kind": "solve", "graph": kind[6:], "n": n, "parts": max(2, n // rng.randint(700, 1100))}
    if kind == "parts":
        n = _log_int(rng, 4000, 24000)
        return {"kind": "parts", "n": n, "parts": max(2, n // rng.randint(700, 1100))}
    if kind == "dropin":
        n = _log_int(rng, 400, 6000)
        return {"kind": "dropin", "n": n, "parts": max(2, n // 800)}
    if kind == "floyd":
        nmax = _log_int(rng, 64, 2048)
        count = max(1, min(512, int(_log_int(rng, 1, 512) * 2048 / nmax)))
        return {"kind": "floyd", "count": count, "nmin": max(16, nmax // rng.randint(1, 64)), "nmax": nmax}
    if kind == "adjoint":
        nmax = _log_int(rng, 64, 1024)
        return {"kind": "adjoint", "count": _log_int(rng, 8, 256), "nmin": max(16, nmax // rng.randint(1, 8)),
                "nmax": nmax, "pairs": _log_int(rng, 500, 20000)}
    if kind.startswith("minplus"):
        m, k = _log_int(rng, 64, 4096), _log_int(rng, 4, 500)
        n = min(_log_int(rng, 256, 120000), (1 << 31) // (m * k) * 4)
        return {"kind": "minplus", "dtype": kind[8:], "m": m, "n": max(n, 256), "k": k}
    if kind == "sssp":
        return {"kind": "sssp", "n": _log_int(rng, 5000, 114599), "sources": _log_int(rng, 1, 200)}
    n = _log_int(rng, 1000, 8000)
    return {"kind": "paths", "n": n, "parts": max(2, n // 1000), "pairs": _log_int(rng, 200, 20000)}


# ---- inputs ---------------------------------------------------------------


def _graph(case, seed):
    family = case.get("graph", "road")
    if family == "grid":
        return graphs.grid_graph(case["rows"], case["cols"], seed=seed)
    if family == "geometric":
        return graphs.geometric_knn(case["n"], seed=seed)
    return graphs.road_like(case["n"], seed=seed)


def _instance_sizes(case):
    """Sizes of a batch's matrices (of the case alone: every seed's batch is the same work)."""
    rng = np.random.default_rng([case["count"], case["nmin"], case["nmax"]])
    lo, hi = case["nmin"], case["nmax"]
    if case["kind"] == "floyd":  # spread over the logarithm, as many small instances as large ones
        s = np.exp(rng.uniform(math.log(lo), math.log(hi + 1), size=case["count"]))
    else:
        s = rng.uniform(lo, hi + 1, size=case["count"])
    return [int(x) for x in np.clip(s, lo, hi)]


def _offsets(sizes):
    """Element offsets of the matrices in one buffer (256-byte aligned, rows dense), and its length."""
    off, acc = [], 0
    for s in sizes:
        off.append(acc)
        acc += (s * s + 63) // 64 * 64
    return off, acc


def _views(flat, off, sizes):
    return [flat[o:o + s * s].view(s, s) for o, s in zip(off, sizes)]


def _instances(case, seed):
    """Input distances and predecessors of a batch in one buffer each."""
    sizes = _instance_sizes(case)
    off, total = _offsets(sizes)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    i32 = case["kind"] == "floyd"
    dist = torch.zeros(total, dtype=torch.int32 if i32 else torch.float32, device="cuda")
    pred = torch.zeros(total, dtype=torch.int32, device="cuda")
    for d, p, s in zip(_views(dist, off, sizes), _views(pred, off, sizes), sizes):
        if i32:  # 5 % of the pairs joined, weights 1..100
            d.fill_(INF_I32)
            edge = torch.rand(s, s, device="cuda", generator=gen) < 0.05
            w = torch.randint(1, 101, (s, s), device="cuda", generator=gen, dtype=torch.int32)
            d.copy_(torch.where(edge, w, d))
            d.fill_diagonal_(0)
            reached = d < INF_I32
        else:  # four edges out of and into every vertex, weights U(0.5, 2)
            d.fill_(INF_F32)
            cols = torch.stack([torch.randperm(s, device="cuda", generator=gen) for _ in range(4)], 1)
            d.scatter_(1, cols, torch.rand(s, 4, device="cuda", generator=gen) * 1.5 + 0.5)
            d.fill_diagonal_(0)
            reached = d < INF_F32
        rows = torch.arange(s, dtype=torch.int32, device="cuda")[:, None]
        p.copy_(torch.where(reached, rows.expand(s, s), torch.full_like(p, -1)))
    return sizes, off, dist, pred


def _pairs(case, seed, sizes):
    """(instance, source, target, gradient) of the adjoint's pairs."""
    rng = np.random.default_rng([seed, 7])
    b = rng.integers(0, len(sizes), size=case["pairs"])
    top = np.asarray(sizes)[b]
    s = (rng.random(case["pairs"]) * top).astype(np.int32)
    t = (rng.random(case["pairs"]) * top).astype(np.int32)
    g = rng.uniform(0.5, 1.5, size=case["pairs"]).astype(np.float32)
    return b.astype(np.int32), s, t, g


def _product(case, seed):
    """A and B of a (min,+) product and B's predecessors; a tenth of the entries unreached."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def side(r, c):
        if case["dtype"] == "f32":
            x = torch.rand(r, c, device="cuda", generator=gen) * 1000.0 + 0.1
        else:
            x = torch.randint(0, 20001, (r, c), device="cuda", generator=gen, dtype=torch.int32)
        gone = torch.rand(r, c, device="cuda", generator=gen) < 0.1
        return x.masked_fill_(gone, INF_F32 if case["dtype"] == "f32" else INF_I32)

    a, b = side(case["m"], case["k"]), side(case["k"], case["n"])
    bp = torch.randint(0, case["n"], b.shape, device="cuda", generator=gen, dtype=torch.int32)
    bp.masked_fill_(b >= (INF_F32 if case["dtype"] == "f32" else INF_I32), -1)
    return a, b, bp


def _sources(case, seed):
    return np.random.default_rng([seed, 3]).permutation(case["n"])[:case["sources"]].astype(np.int32)


def _path_pairs(case, seed):
    rng = np.random.default_rng([seed, 5])
    s, t = (rng.integers(0, case["n"], size=case["pairs"]).astype(np.int32) for _ in range(2))
    return s, t, rng.uniform(0.5, 1.5, size=case["pairs"]).astype(np.float32)


MAX_PATH = 512  # path slots per query


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "parts", "dropin", "sssp", "paths"):
        g = _graph(case, seed)
        if kind == "sssp":
            gid = np.ones(g.n, np.int32)  # one part: only the graph itself is searched
            parts = 1
        else:
            parts = case["parts"]
            gid, _ = fap.partition(g.row_offset, g.col_val, parts)
        if kind == "dropin":
            fg = fap.FapGraph(g.n, g.m, g.row_offset, g.col_val, g.weight, parts, graph_id=gid)
            fg.preCondition()
            return {"kind": kind, "graph": fg}
        integer = case.get("graph") in ("grid", "geometric")
        eng = fap.Engine(g.n, g.row_offset, g.col_val, g.weight, parts, graph_id=gid,
                         dtype=fap.DTYPE_I32 if integer else fap.DTYPE_F32)
        dtype = torch.int32 if integer else torch.float32
        if kind == "solve" and not integer:
            eng.set_option(fap._lib.OPT_SSSP_FP64, 1)  # boundary rows exact, rounded once
        rows = case["sources"] if kind == "sssp" else g.n
        state = {"kind": kind, "engine": eng,
                 "dist": torch.empty((rows, g.n), dtype=dtype, device="cuda"),
                 "pred": torch.empty((rows, g.n), dtype=torch.int32, device="cuda")}
        if kind == "parts":
            state["spans"] = [(p, eng.part_info(p)[2], eng.part_info(p)[0]) for p in range(1, parts + 1)]
        elif kind == "sssp":
            state["sources"] = _sources(case, seed)
        elif kind == "paths":
            eng.solve(state["dist"], state["pred"])  # the rows that the queries read
            s, t, w = _path_pairs(case, seed)
            nq = s.shape[0]
            state.update(stream=torch.cuda.Stream(), s=torch.from_numpy(s).cuda(), t=torch.from_numpy(t).cuda(),
                         g=torch.from_numpy(w).cuda(),
                         out_dist=torch.empty(nq, device="cuda"),
                         out_len=torch.empty(nq, dtype=torch.int32, device="cuda"),
                         out_path=torch.full((nq, MAX_PATH), -1, dtype=torch.int32, device="cuda"),
                         dw=torch.zeros(g.m, device="cuda"))
        return state
    # the program's own stream: the kernels run behind what it queued there
    state = {"kind": kind, "ctx": fap.Context(), "stream": torch.cuda.Stream()}
    if kind == "minplus":
        a, b, bp = _product(case, seed)
        state.update(dtype=fap.DTYPE_F32 if case["dtype"] == "f32" else fap.DTYPE_I32, a=a, b=b, bp=bp,
                     c=torch.empty((case["m"], case["n"]), dtype=a.dtype, device="cuda"),
                     cp=torch.empty((case["m"], case["n"]), dtype=torch.int32, device="cuda"))
        return state
    sizes, off, dist, pred = _instances(case, seed)
    d, p = torch.zeros_like(dist), torch.zeros_like(pred)
    state.update(dtype=fap.DTYPE_I32 if kind == "floyd" else fap.DTYPE_F32, dist0=dist, pred0=pred, dist=d, pred=p,
                 mats=_views(d, off, sizes), preds=_views(p, off, sizes))
    if kind == "adjoint":
        dw = torch.zeros_like(d)
        state.update(dw=dw, dws=_views(dw, off, sizes),
                     pairs=[torch.from_numpy(x).cuda() for x in _pairs(case, seed, sizes)])
    return state


# ---- one pass -------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "solve":
        state["engine"].solve(state["dist"], state["pred"], fap.MODE_BATCHED)
        return {"dist": state["dist"], "pred": state["pred"]}
    if kind == "parts":
        for part, first, rows in state["spans"]:
            state["engine"].solve_part(part, state["dist"][first:first + rows], state["pred"][first:first + rows])
        return {"dist": state["dist"], "pred": state["pred"]}
    if kind == "dropin":
        fg = state["graph"]
        fg.solve()
        return {"dist": fg.getAllDistance(), "pred": fg.getAllPath()}
    if kind == "sssp":
        state["engine"].sssp(state["sources"], state["dist"], state["pred"])
        return {"dist": state["dist"], "pred": state["pred"]}
    stream = state["stream"]
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        if kind == "paths":
            eng = state["engine"]
            eng.query(state["dist"], state["pred"], state["s"], state["t"], state["out_dist"], state["out_len"],
                      state["out_path"], MAX_PATH, stream=stream.cuda_stream)
            state["dw"].zero_()
            eng.backward(state["pred"], state["s"], state["t"], state["g"], state["dw"], stream=stream.cuda_stream)
            return {"dist": state["out_dist"], "len": state["out_len"], "path": state["out_path"], "dw": state["dw"]}
        if kind == "minplus":
            state["ctx"].minplus(state["dtype"], state["a"], state["b"], state["c"], Bp=state["bp"], Cp=state["cp"],
                                 stream=stream.cuda_stream)
            return {"dist": state["c"], "pred": state["cp"]}
        state["dist"].copy_(state["dist0"])  # the closure is in place
        state["pred"].copy_(state["pred0"])
        state["ctx"].floyd_batched(state["dtype"], state["mats"], state["preds"], stream=stream.cuda_stream)
        if kind == "floyd":
            return {"dist": state["dist"], "pred": state["pred"]}
        state["dw"].zero_()
        b, s, t, g = state["pairs"]
        state["ctx"].backward_dense(state["preds"], state["dws"], b, s, t, g, stream=stream.cuda_stream)
        return {"dist": state["dist"], "pred": state["pred"], "dw": state["dw"]}


# ---- what a pass cannot do without ------------------------------------------


def work(case):
    kind = case["kind"]
    if kind in ("solve", "parts", "dropin", "paths"):
        n = case["rows"] * case["cols"] if case.get("graph") == "grid" else case["n"]
        if kind == "paths":  # the walks: their lengths are the graph's, taken as its side
            steps = case["pairs"] * math.sqrt(n)
            return {"bytes": 8.0 * steps + 16.0 * case["pairs"], "flops": steps}
        # rows of distances and predecessors, and the closure of every part (one add and one minimum a step)
        return {"bytes": 8.0 * n * n + 24.0 * n, "flops": 2.0 * case["parts"] * (n / case["parts"]) ** 3}
    if kind == "sssp":
        return {"bytes": 8.0 * case["sources"] * case["n"] + 21.0 * case["n"],
                "flops": 2.0 * case["sources"] * 2.1 * case["n"]}
    if kind == "minplus":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4.0 * m * k + 8.0 * k * n + 8.0 * m * n, "flops": 2.0 * m * n * k}
    sizes = np.asarray(_instance_sizes(case), np.float64)
    area = float((sizes ** 2).sum())
    # matrices read and written; the input copy that an in-place closure needs; the gradient's zeros
    return {"bytes": area * (16.0 if kind == "floyd" else 20.0), "flops": 2.0 * float((sizes ** 3).sum())}


# ---- the same in 64 bits ------------------------------------------------------


def _relax64(g, sources):
    """FP64 distances from `sources` (rows) by relaxing every in-edge until nothing changes."""
    n = g.n
    src = np.repeat(np.arange(n), np.diff(g.row_offset))
    order = np.argsort(g.col_val, kind="stable")
    dst, src, w = g.col_val[order], src[order], g.weight[order].astype(np.float64)
    deg = np.bincount(dst, minlength=n)
    width = int(deg.max())
    slot = np.arange(dst.shape[0]) - np.repeat(np.cumsum(deg) - deg, deg)
    nb = np.tile(np.arange(n)[:, None], (1, width))  # padding: the vertex itself at weight 0
    wt = np.zeros((n, width))
    nb[dst, slot], wt[dst, slot] = src, w
    nb, wt = torch.from_numpy(nb).cuda(), torch.from_numpy(wt).cuda()
    out = torch.empty((len(sources), n), dtype=torch.float64, device="cuda")
    for c in range(0, len(sources), 4096):
        some = torch.as_tensor(np.asarray(sources[c:c + 4096]), device="cuda").long()
        d = torch.full((n, some.shape[0]), math.inf, dtype=torch.float64, device="cuda")
        d[some, torch.arange(some.shape[0], device="cuda")] = 0.0
        for it in range(1, n + 1):
            new = d
            for j in range(width):
                new = torch.minimum(new, d[nb[:, j]] + wt[:, j:j + 1])
            if it % 16 == 0 and torch.equal(new, d):
                break
            d = new
        out[c:c + 4096] = d.t()
    return out


def _pred64(g, dist):
    """Predecessors of FP64 rows (row s: source s): the in-neighbour whose edge is tight."""
    src = torch.from_numpy(np.repeat(np.arange(g.n), np.diff(g.row_offset))).cuda()
    dst = torch.from_numpy(g.col_val.astype(np.int64)).cuda()
    w = torch.from_numpy(g.weight.astype(np.float64)).cuda()
    pred = torch.full(dist.shape, -1, dtype=torch.int64, device="cuda")
    edge = torch.full(dist.shape, -1, dtype=torch.int64, device="cuda")
    for e in range(0, src.shape[0], 1024):
        u, v, x = src[e:e + 1024], dst[e:e + 1024], w[e:e + 1024]
        tight = (dist[:, u] + x <= dist[:, v] * (1 + 1e-13)) & torch.isfinite(dist[:, v])
        r, i = tight.nonzero(as_tuple=True)
        pred[r, v[i]] = u[i]
        edge[r, v[i]] = e + i
    return pred, edge


def exact(case, seed):
    kind = case["kind"]
    if kind == "floyd" or (kind == "solve" and case["graph"] != "road") or \
            (kind == "minplus" and case["dtype"] == "i32"):
        return None  # whole numbers
    if kind == "minplus":
        a, b, _ = (x.double() for x in _product(case, seed))
        a[a >= INF_F32] = math.inf
        b[b >= INF_F32] = math.inf
        c = torch.full((case["m"], case["n"]), math.inf, dtype=torch.float64, device="cuda")
        for k in range(case["k"]):
            torch.minimum(c, a[:, k:k + 1] + b[k:k + 1], out=c)
        return {"dist": c.nan_to_num(posinf=INF_F32), "pred": None}
    if kind == "adjoint":
        sizes, off, dist, pred = _instances(case, seed)
        top = max(sizes)
        d = torch.full((len(sizes), top, top), math.inf, dtype=torch.float64, device="cuda")
        p = torch.full((len(sizes), top, top), -1, dtype=torch.int32, device="cuda")
        for i, (x, q, s) in enumerate(zip(_views(dist, off, sizes), _views(pred, off, sizes), sizes)):
            d[i, :s, :s] = torch.where(x < INF_F32, x.double(), math.inf)
            p[i, :s, :s] = q
        for k in range(top):
            via = d[:, :, k:k + 1] + d[:, k:k + 1, :]
            better = via < d
            torch.where(better, p[:, k:k + 1, :].expand_as(p), p, out=p)
            torch.minimum(d, via, out=d)
        dw = torch.zeros_like(d)
        b, s, t, g = (torch.from_numpy(x).cuda() for x in _pairs(case, seed, sizes))
        b, s, v, g = b.long(), s.long(), t.long(), g.double()
        g = torch.where(torch.isfinite(d[b, s, v]), g, 0.0)
        for _ in range(top):
            live = (v != s) & (g != 0)
            if not bool(live.any()):
                break
            b, s, v, g = b[live], s[live], v[live], g[live]
            u = p[b, s, v].long()
            dw.index_put_((b, u, v), g, accumulate=True)
            v = u
        flat = [torch.zeros(dist.shape, dtype=torch.float64, device="cuda") for _ in range(2)]
        for i, s in enumerate(sizes):
            for f, x in zip(flat, (d, dw)):
                f[off[i]:off[i] + s * s] = x[i, :s, :s].nan_to_num(posinf=INF_F32).reshape(-1)
        return {"dist": flat[0], "pred": None, "dw": flat[1]}
    if kind != "sssp" and case["n"] > 25000:
        return None  # the relaxation over all sources takes longer than is wanted
    g = _graph(case, seed)
    if kind == "sssp":
        return {"dist": _relax64(g, _sources(case, seed)).nan_to_num(posinf=INF_F32), "pred": None}
    if kind == "paths":
        d = _relax64(g, np.arange(g.n))
        s, t, w = (torch.from_numpy(x).cuda() for x in _path_pairs(case, seed))
        s, v, w = s.long(), t.long(), w.double()
        reached = d[s, v].nan_to_num(posinf=INF_F32)
        pred, edge = _pred64(g, d)
        w = torch.where(torch.isfinite(d[s, v]), w, 0.0)
        dw = torch.zeros(g.m, dtype=torch.float64, device="cuda")
        for _ in range(g.n):
            live = (v != s) & (w != 0)
            if not bool(live.any()):
                break
            s, v, w = s[live], v[live], w[live]
            dw.index_put_((edge[s, v],), w, accumulate=True)
            v = pred[s, v]
        return {"dist": reached, "len": None, "path": None, "dw": dw}
    gid, _ = fap.partition(g.row_offset, g.col_val, case["parts"])
    order = fap.preprocess(case["parts"], gid, g.row_offset, g.col_val)["st2ed"]  # the rows' order
    d = _relax64(g, order).nan_to_num(posinf=INF_F32)
    return {"dist": d if kind != "dropin" else d.cpu().numpy(), "pred": None}
