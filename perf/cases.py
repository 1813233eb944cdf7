"""The framework's workloads, for measuring it: decompositions with their
densest search from the smallest to the largest graphs, one graph from host
memory to host results, batches, serving, and queries on a finished table.

A case is a dict of plain values.  ``do`` names the call sequence:

* ``grid``: the core table into a device tensor, then the densest search for
  every value of ``betas``, on a graph resident on the device;
* ``fresh``: the same from the host graph to pinned host memory, upload
  included;
* ``batch``: many graphs in one batched call;
* ``serve``: a burst of requests to a server, graphs resident;
* ``cells``: the table and every cell as a prefix of one order per column;
* ``members``: many cells' node sets from a resident table.

Graphs are Chung-Lu (``gamma`` > 0: n nodes, L layers of n * degree / 2 edges,
a ``copy`` share of them taken from layer 0) or Erdos-Renyi layers
(``gamma`` = 0: p uniform in [p_lo, p_hi]); every node has at least one edge,
as in a loaded graph, so a case's shapes do not depend on its seed.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import pargridcpu_b200 as fc
from pargridcpu_b200 import native

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _cl(do, n, L, degree, gamma, copy, **more):
    return dict(do=do, n=n, L=L, degree=degree, gamma=gamma, copy=copy, **more)


def listed():
    return [
        dict(_cl("grid", 1000, 2, 4.0, 2.5, 0.3, betas="1"), name="small"),
        dict(_cl("grid", 20_000, 7, 2.0, 2.5, 0.3, betas="1"), name="plain 20k x 7"),
        dict(do="grid", n=220, L=360, degree=0.0, gamma=0.0, copy=0.0, p_lo=0.01, p_hi=0.06,
             betas="1", name="layers 220 x 360"),
        dict(_cl("grid", 45_003, 13, 8.0, 2.5, 0.3, betas="1"), name="middle 45k x 13"),
        dict(_cl("grid", 180_001, 17, 24.0, 2.4, 0.25, betas="1"), name="dense 180k x 17"),
        dict(_cl("grid", 2_500_000, 4, 6.8, 2.1, 0.5, betas="0.5,1,2"), name="hubs 2.5M x 4"),
        dict(_cl("grid", 2_600_000, 24, 2_000_000 / 1_300_000, 2.2, 0.4, betas="1"),
             name="wide 2.6M x 24"),
        dict(_cl("fresh", 1_250_001, 4, 6.8, 2.1, 0.5, betas="1"), name="fresh 1.25M x 4"),
        dict(do="batch", graphs=24, mix=404, n_lo=1_000, n_hi=100_000, betas="1", name="batch 24"),
        dict(do="serve", graphs=8, mix=505, n_lo=1_000, n_hi=60_000, betas="1", requests=12,
             name="serve 12"),
        dict(_cl("cells", 120_000, 9, 6.0, 2.3, 0.3), name="cells 120k x 9"),
        dict(_cl("members", 300_001, 10, 8.0, 2.4, 0.3, queries=32, by_index=False),
             name="members 300k x 10"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _drawn_graph(rng, n_lo, n_hi):
    n, L = int(_log(rng, n_lo, n_hi)), rng.randint(1, 24)
    return dict(n=n, L=L, degree=round(min(_log(rng, 2, 32), 9e7 / (n * L)), 3),
                gamma=round(rng.uniform(2.0, 3.0), 3), copy=round(rng.uniform(0, 0.6), 3))


def draw(rng):
    betas = rng.choice(["1", "1", "0.5,1,2", "0.5"])
    t = rng.random()
    if t < 0.1:
        return dict(do="grid", n=rng.randint(100, 400), L=rng.randint(33, 380), degree=0.0,
                    gamma=0.0, copy=0.0, p_lo=0.01, p_hi=round(rng.uniform(0.03, 0.08), 4),
                    betas=betas)
    if t < 0.25:
        return dict(do="batch", graphs=rng.randint(4, 32), mix=rng.randrange(1 << 20), n_lo=1_000,
                    n_hi=int(_log(rng, 20_000, 100_000)), betas="1")
    if t < 0.35:
        return dict(do="serve", graphs=rng.randint(2, 8), mix=rng.randrange(1 << 20), n_lo=1_000,
                    n_hi=int(_log(rng, 20_000, 60_000)), betas="1", requests=rng.randint(2, 16))
    if t < 0.45:
        return dict(do="members", queries=rng.randint(1, 64), by_index=rng.random() < 0.5,
                    **_drawn_graph(rng, 1_000, 300_000))
    if t < 0.55:
        return dict(do="cells", **_drawn_graph(rng, 1_000, 300_000))
    do = "fresh" if t < 0.7 else "grid"
    return dict(do=do, betas=betas, **_drawn_graph(rng, 1_000, 1_500_000))


# ---- graphs --------------------------------------------------------------------

def _unique_fill(drawer, base, target, gen):
    """``base`` (sorted, distinct) plus fresh distinct draws, ``target`` in all."""
    s = base
    while len(s) < target:
        s = torch.unique(torch.cat([s, drawer(int((target - len(s)) * 1.3) + 64)]))
    if len(s) > target:
        fresh = s[~torch.isin(s, base, assume_unique=True)]
        keep = torch.randperm(len(fresh), generator=gen, device=DEV)[:target - len(base)]
        s = torch.sort(torch.cat([base, fresh[keep]])).values
    return s


def _layers(case, seed):
    """Per layer the distinct undirected edges, as sorted keys u * n + v, u < v."""
    n, L = case["n"], case["L"]
    gen = torch.Generator(device=DEV).manual_seed(seed * 7919 + n * 31 + L)
    empty = torch.empty(0, dtype=torch.int64, device=DEV)
    if not case["gamma"]:
        iu = torch.triu_indices(n, n, 1, device=DEV)
        every = iu[0] * n + iu[1]
        p = random.Random(n * 1009 + L)
        out = [every[torch.rand(len(every), generator=gen, device=DEV) <
                     p.uniform(case["p_lo"], case["p_hi"])] for _ in range(L)]
        ends = torch.arange(n, device=DEV)
        mate = torch.randint(n, (n,), generator=gen, device=DEV)
    else:
        w = torch.arange(1, n + 1, dtype=torch.float64, device=DEV) ** (-1 / (case["gamma"] - 1))
        cdf = torch.cumsum(w, 0)
        cdf /= cdf[-1].clone()
        label = torch.randperm(n, generator=gen, device=DEV)

        def ends_of(k):
            at = torch.searchsorted(cdf, torch.rand(k, generator=gen, device=DEV,
                                                    dtype=torch.float64), right=True)
            return label[at.clamp_(max=n - 1)]

        def drawer(k):
            a, b = ends_of(k), ends_of(k)
            key = torch.minimum(a, b) * n + torch.maximum(a, b)
            return key[a != b]

        m = max(1, min(int(n * case["degree"] / 2), n * (n - 1) // 2))
        out = [_unique_fill(drawer, empty, m, gen)]
        for _ in range(L - 1):
            pick = torch.randperm(m, generator=gen, device=DEV)[:int(case["copy"] * m)]
            base = torch.sort(out[0][pick]).values
            out.append(_unique_fill(drawer, base, m, gen))
        mate = ends_of(n)
    # a node without edges gets one, in a layer of its own
    seen = torch.zeros(n, dtype=torch.bool, device=DEV)
    for key in out:
        seen[key // n] = True
        seen[key % n] = True
    lone = torch.nonzero(~seen).reshape(-1)
    if len(lone):
        to = mate[lone]
        to = torch.where(to == lone, (lone + 1) % n, to)
        key = torch.minimum(lone, to) * n + torch.maximum(lone, to)
        for l in range(L):
            more = key[lone % L == l]
            if len(more):
                out[l] = torch.unique(torch.cat([out[l], more]))
    return out


def _graph(case, seed):
    """The graph in the reference's in-memory form ([deg, nbrs...] rows)."""
    n = case["n"]
    bufs = []
    for key in _layers(case, seed):
        a, b = key // n, key % n
        both = torch.sort(torch.cat([a * n + b, b * n + a])).values
        src, dst = both // n, both % n
        deg = torch.bincount(src, minlength=n)
        at = torch.cumsum(deg, 0) - deg + torch.arange(n, device=DEV)
        buf = torch.empty(n + len(both), dtype=torch.int32, device=DEV)
        buf[at] = deg.to(torch.int32)
        buf[torch.arange(len(both), device=DEV) + src + 1] = dst.to(torch.int32)
        bufs.append(buf.cpu().numpy().view(np.uint32))
    return fc.MultilayerGraph.from_adjbuf(n, bufs)


def _mix(case):
    """The graphs of a batch: sizes from the case alone, edges from the seed."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["graphs"]):
        n = int(_log(r, case["n_lo"], case["n_hi"]))
        out.append(dict(n=n, L=r.randint(2, 24), degree=_log(r, 2, 32), gamma=r.uniform(2, 3),
                        copy=r.uniform(0, 0.6)))
    return out


def _betas(case):
    return [float(b) for b in case["betas"].split(",")]


def prepare(case, seed):
    do = case["do"]
    s = {"case": case}
    if do in ("batch", "serve"):
        s["graphs"] = [_graph(c, seed * 97 + i) for i, c in enumerate(_mix(case))]
        for g in s["graphs"]:
            g.upload()
        if do == "serve":
            s["server"] = fc.Server()
        return s
    n, L = case["n"], case["L"]
    g = s["g"] = _graph(case, seed)
    if do == "fresh":
        table = torch.empty((L, n), dtype=torch.int32, pin_memory=DEV == "cuda")
        s["table"] = table.numpy().view(np.uint32)
        return s
    g.upload()
    s["table"] = torch.empty((L, n), dtype=torch.int32, device=DEV)
    if do == "cells":
        s["order"] = np.zeros((L, n), np.uint32)
        s["off"] = np.zeros(L + 1, np.uint64)
        s["sizes"] = np.zeros(L * 4096, np.uint32)
    if do == "members":
        r, q = random.Random(seed), case["queries"]
        s["ks"] = np.array([r.randint(1, 12) for _ in range(q)], np.uint32)
        s["lmds"] = np.array([r.randint(1, L) for _ in range(q)], np.uint32)
        s["off"] = np.zeros(q + 1, np.uint64)
        s["nodes"] = np.zeros(q * n, np.uint32)
        g.coreindex(copy=False)
    return s


def _results(res):
    whole = ("k", "lmd", "length", "lstar", "n_cells")
    return {"cell": np.array([[r[f] for f in whole] for r in res], np.int64),
            "density": np.array([r["density"] for r in res], np.float64)}


def run(s):
    case, do = s["case"], s["case"]["do"]
    if do == "grid":
        g = s["g"]
        g.reset_results()
        g.coreindex(out=s["table"])
        return dict(table=s["table"], **_results(g.densest(_betas(case))))
    if do == "fresh":
        g = s["g"]
        g.release_device()
        table, res = g.coreindex_densest(out=s["table"], betas=_betas(case))
        return dict(table=table.view(np.int32), **_results(res))
    if do == "batch":
        tables, res, _ = fc.batch_run(s["graphs"], beta=_betas(case)[0])
        return dict(tables=[t.view(np.int32) for t in tables], **_results(res))
    if do == "serve":
        sv, gs = s["server"], s["graphs"]
        tickets = [sv.submit(gs[i % len(gs)], beta=_betas(case)[0])
                   for i in range(case["requests"])]
        done = [sv.wait(t) for t in tickets]
        return dict(tables=[t.view(np.int32) for t, _, _ in done],
                    **_results([r for _, r, _ in done]))
    lib, cnt = native.lib(), C.c_uint64()
    if do == "cells":
        g = s["g"]
        g.reset_results()
        g.coreindex(out=s["table"])
        native.check(lib.fc_cell_index(g.handle, native.ptr(s["order"]), native.ptr(s["off"]),
                                       native.ptr(s["sizes"]), len(s["sizes"]), C.byref(cnt), None),
                     "cell_index")
        return {"table": s["table"], "order": s["order"].view(np.int32),
                "off": s["off"].view(np.int64), "sizes": s["sizes"].view(np.int32)}
    native.check(lib.fc_cells_members(s["g"].handle, native.ptr(s["ks"]), native.ptr(s["lmds"]),
                                      len(s["ks"]), int(case["by_index"]), native.ptr(s["off"]),
                                      native.ptr(s["nodes"]), len(s["nodes"]), None),
                 "cells_members")
    return {"off": s["off"].view(np.int64), "nodes": s["nodes"].view(np.int32)}


def _sizes(c):
    """(nodes, layers, directed entries) of one graph, expected."""
    if not c["gamma"]:
        return c["n"], c["L"], int(c["n"] ** 2 * c["L"] * (c["p_lo"] + c["p_hi"]) / 2)
    return c["n"], c["L"], 2 * c["L"] * max(1, min(int(c["n"] * c["degree"] / 2),
                                                   c["n"] * (c["n"] - 1) // 2))


def work(case):
    do = case["do"]
    if do == "members":  # every queried column read, its offsets and about half the ids written
        return {"bytes": case["queries"] * (4 * case["n"] + 2 * case["n"] + 8), "flops": 0}
    if do in ("batch", "serve"):
        graphs = _mix(case)
        if do == "serve":  # repeated requests of one graph return its table again
            graphs = [graphs[i % len(graphs)] for i in range(case["requests"])]
    else:
        graphs = [case]
    total = 0
    for n, L, e in map(_sizes, graphs):
        total += 4 * e + 4 * (n + 1) + 4 * n * L      # the rows, once, and the table
        total += 4 * n * L if do == "cells" else 0     # the order
        total += 4 * L * (n + 1) if do == "fresh" else 0
    return {"bytes": total, "flops": 0}


# ---- the same in plain torch ------------------------------------------------------

def _table64(n, L, src, dst, layer):
    """core_lambda(v) for every lambda, by peeling level by level."""
    deg0 = torch.bincount(src * L + layer, minlength=n * L).reshape(n, L)
    table = torch.zeros((L, n), dtype=torch.int64, device=DEV)
    for lam in range(1, L + 1):
        deg, alive, k = deg0.clone(), torch.ones(n, dtype=torch.bool, device=DEV), 0
        while True:
            top = torch.topk(deg, lam, dim=1).values[:, -1]
            top = torch.where(alive, top, torch.iinfo(torch.int64).max)
            low = int(top.min())
            if low == torch.iinfo(torch.int64).max:
                break
            k = max(k, low)
            gone = top <= k
            table[lam - 1][gone] = k
            alive &= ~gone
            e = gone[src]
            deg -= torch.bincount(dst[e] * L + layer[e], minlength=n * L).reshape(n, L)
    return table


def exact(case, seed):
    if case["do"] not in ("grid", "fresh"):
        return None
    n, L, e = _sizes(case)
    if e * L > 3e8:
        return None
    keys = _layers(case, seed)
    a = torch.cat([k // n for k in keys] + [k % n for k in keys])
    b = torch.cat([k % n for k in keys] + [k // n for k in keys])
    layer = torch.cat([torch.full_like(k, l) for l, k in enumerate(keys)] * 2)
    table = _table64(n, L, a, b, layer)
    best = [0.0] * len(_betas(case))
    power = [torch.arange(1, L + 1, dtype=torch.float64, device=DEV) ** x for x in _betas(case)]
    for lam in range(L):
        core = table[lam]
        kmax = int(core.max())
        if not kmax:
            continue
        key = torch.minimum(core[a], core[b])
        hist = torch.bincount(key * L + layer, minlength=(kmax + 1) * L).reshape(kmax + 1, L)
        ends = torch.flip(torch.cumsum(torch.flip(hist, [0]), 0), [0])[1:]  # k = 1 .. kmax
        size = torch.flip(torch.cumsum(torch.flip(torch.bincount(core), [0]), 0), [0])[1:]
        dens = torch.sort(ends, dim=1, descending=True).values.double() / 2 / size.double()[:, None]
        for i, p in enumerate(power):
            best[i] = max(best[i], float((dens * p).max()))
    return {"table": None, "cell": None, "density": np.array(best, np.float64)}
