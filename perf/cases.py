"""Performance cases: evaluations of ASPL and diameter as programs run them.

A case is one call (or one round of calls) of a program that keeps its plan,
server or chains and evaluates graphs that live in host memory:

  general, grid   ODP_Init_aspl_* once, then ODP_Set_aspl per graph: the loop
                  of an optimiser that proposes one graph after another
  batch           a plan over many graphs of uneven size, degree and symmetry
                  (a population, a parameter sweep), run on new adjacencies
  serve           resident graphs on a server; one round submits a 2-opt move
                  of every chain and waits for all results
  anneal          simulated-annealing chains whose steps run on the GPU; one
                  pass is a number of steps and the read-back of all chains

Random general graphs are drawn from the configuration model (with its
cyclic lifts for symmetries > 1), grid graphs by local 2-opt swaps of a
folded lattice: the graphs such programs start from and move through.
"""
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import odp_gb300 as og
from odp_gb300 import workloads


def listed():
    return [
        # The smallest published problem sizes, where only launches and latency count.
        dict(name="general n256 d5", kind="general", n=256, d=5, s=1, irregular=False),
        # The README's annealing example, one call per proposal.
        dict(name="general n1024 d8", kind="general", n=1024, d=8, s=1, irregular=False),
        # An ordinary dense graph of a few thousand vertices.
        dict(name="general n4096 d24", kind="general", n=4096, d=24, s=1, irregular=False),
        # Odd size, odd symmetry, vertices of different degrees.
        dict(name="general n9999 d12 s3 irregular", kind="general", n=9999, d=12, s=3, irregular=True),
        # The large single graph of the benchmark.
        dict(name="general n65536 d16", kind="general", n=65536, d=16, s=1, irregular=False),
        # The benchmark's symmetric graph: many rows, few sources.
        dict(name="general n262144 d24 s64", kind="general", n=262144, d=24, s=64, irregular=False),
        # A grid as small as the published ones, tens of short levels.
        dict(name="grid 50x50 d4 l3", kind="grid", w=50, h=50, d=4, length=3),
        # A mid-size grid with odd, unequal sides.
        dict(name="grid 97x103 d6 l4", kind="grid", w=97, h=103, d=6, length=4),
        # The largest grid of the tests and the benchmark.
        dict(name="grid 256x256 d6 l4", kind="grid", w=256, h=256, d=6, length=4),
        # The benchmark's batch of uneven graphs, half as many of them.
        dict(name="batch 256 mixed", kind="batch", count=256, n_lo=256, n_hi=8192, draw_seed=100),
        # The served annealing chains that fit a low-latency service.
        dict(name="serve 32 chains", kind="serve", chains=32, n_lo=1024, n_hi=4096, d=16),
        # A group of equal chains annealing on the GPU.
        dict(name="anneal 16 chains n1024 d8", kind="anneal", chains=16, n=1024, d=8, steps=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["general", "general", "general", "grid", "grid", "grid", "batch", "serve", "anneal"])
    if kind == "general":
        s = rng.choice([1, 1, 1, 2, 3, 4, 16])
        n = _log_int(rng, 64, 65536) // s * s
        d = rng.randint(3, 24)
        if n // s * d % 2:
            d += 1
        return dict(kind=kind, n=n, d=d, s=s, irregular=rng.random() < 0.2)
    if kind == "grid":
        w, h = _log_int(rng, 10, 200), _log_int(rng, 10, 200)
        return dict(kind=kind, w=w, h=h, d=2 * rng.randint(2, 5), length=rng.randint(3, 6))
    if kind == "batch":
        lo = _log_int(rng, 64, 1024)
        return dict(kind=kind, count=_log_int(rng, 2, 200), n_lo=lo, n_hi=lo * rng.randint(2, 8),
                    draw_seed=rng.randint(1, 10000))
    if kind == "serve":
        lo = _log_int(rng, 256, 2048)
        return dict(kind=kind, chains=_log_int(rng, 1, 48), n_lo=lo, n_hi=lo * rng.randint(1, 3),
                    d=2 * rng.randint(2, 12))
    return dict(kind=kind, chains=_log_int(rng, 1, 32), n=_log_int(rng, 64, 4096), d=2 * rng.randint(2, 8),
                steps=rng.randint(4, 64))


# --------------------------------------------------------------------------
# Graphs.
# --------------------------------------------------------------------------

def general_adjacency(n, d, s, gen, degrees=None):
    """Compact adjacency int32[n/s][d] of a random graph, d-regular or with
    the given degrees: stubs of the n/s base vertices paired at random, each
    edge with a random rotation."""
    base = n // s
    degrees = np.full(base, d) if degrees is None else degrees
    stubs = np.repeat(np.arange(base, dtype=np.int64), degrees)
    gen.shuffle(stubs)
    a, b = stubs[0::2].copy(), stubs[1::2].copy()
    if s == 1:
        for i in np.flatnonzero(a == b):              # no loops: swap with another edge's end
            while a[i] == b[i]:
                j = int(gen.integers(len(a)))
                if a[j] != b[i] and b[j] != a[i]:
                    b[i], b[j] = b[j], b[i]
    t = gen.integers(0, s, len(a))
    t = np.where((a == b) & (t == 0) & (s > 1), 1, t)
    src = np.concatenate([a, b])
    dst = np.concatenate([(b + t * base) % n, (a + (s - t) * base) % n])
    adj = np.full((base, d), -1, dtype=np.int32)
    adj[np.arange(d)[None, :] < degrees[:, None]] = dst[np.argsort(src, kind="stable")]
    return adj


def _ring(k):
    """Vertices of 0..k-1 in ring order, neighbours at most 2 apart."""
    return np.concatenate([np.arange(0, k, 2), np.arange(1, k, 2)[::-1]])


def _rotate(v, w, h, s, steps=1):
    """Vertices v turned by `steps` of the grid symmetry s (180 or 90 degrees each)."""
    x, y = v // h, v % h
    for _ in range(steps):
        x, y = (w - 1 - x, h - 1 - y) if s == 2 else (y, h - 1 - x)
    return x * h + y


def _base_vertices(w, h, s):
    """The vertex of each row of the compact adjacency."""
    m = np.arange(w * h // s)
    return m if s != 4 else (m // (h // 2)) * h + m % (h // 2)


def grid_adjacency(w, h, d, length, gen, s=1):
    """Compact adjacency int32[w*h/s][d] (d even; a multiple of 4 for s = 4)
    of a grid graph with edges at most `length` long: folded rings along both
    axes, then rounds of 2-opt swaps between edges that start close together.
    With symmetry s an edge stands for its orbit, and both ends of a swap are
    turned together."""
    n = w * h
    vid = np.arange(n).reshape(w, h)
    ends = []
    for k in range(d // 2):                            # ring neighbours at distance 1, then 2 (2 or 4 apart)
        axis, hop = k % 2, min(k // 2 + 1, max(1, length // 2))
        v = vid[_ring(w)] if axis == 0 else vid[:, _ring(h)]
        ends.append(np.stack([v.ravel(), np.roll(v, -hop, axis=axis).ravel()]))
    u, v = np.concatenate(ends, axis=1)
    if s > 1:                                          # one edge of each orbit (parallel edges stay parallel)
        turned = [(_rotate(u, w, h, s, t), _rotate(v, w, h, s, t)) for t in range(s)]
        keys = np.stack([np.minimum(a, b) * n + np.maximum(a, b) for a, b in turned])
        order = np.argsort(keys.min(axis=0), kind="stable")[::s]
        u, v = u[order], v[order]
    m = len(u)
    for _ in range(24):
        flip = gen.random(m) < 0.5
        u, v = np.where(flip, v, u), np.where(flip, u, v)
        if s > 1:
            turn = gen.integers(0, s, m)
            u, v = (np.choose(turn, [_rotate(z, w, h, s, t) for t in range(s)]) for z in (u, v))
        cx, cy = gen.integers(0, length, 2)
        cell = (u // h + cx) // length * (h + 2 * length) + (u % h + cy) // length
        order = np.lexsort((gen.random(m), cell))
        i, j = order[:-1:2], order[1::2][:len(order[:-1:2])]
        far = np.maximum(abs(u[i] // h - v[j] // h) + abs(u[i] % h - v[j] % h),
                         abs(u[j] // h - v[i] // h) + abs(u[j] % h - v[i] % h))
        ok = (cell[i] == cell[j]) & (far <= length) & (u[i] != v[j]) & (u[j] != v[i])
        if s > 1:                                      # no edge that is its own image
            half = _rotate(v, w, h, s, s // 2)
            ok &= (u[i] != half[j]) & (u[j] != half[i])
        i, j = i[ok], j[ok]
        v[i], v[j] = v[j], v[i]
    src = np.concatenate([_rotate(z, w, h, s, t) for t in range(s) for z in (u, v)])
    dst = np.concatenate([_rotate(z, w, h, s, t) for t in range(s) for z in (v, u)])
    full = dst[np.argsort(src, kind="stable")].reshape(n, d).astype(np.int32)
    return np.ascontiguousarray(full[_base_vertices(w, h, s)])


def _degrees(case):
    """The degree table that an irregular case keeps over all its graphs."""
    if not case.get("irregular"):
        return None
    v = np.arange(case["n"] // case["s"], dtype=np.int64)
    return (case["d"] - 2 * ((v * 2654435761 >> 9) % 3 == 0)).astype(np.int32)


def _graph(case, seed):
    """The compact adjacency of a general or grid case."""
    gen = np.random.default_rng(seed)
    if case["kind"] == "grid":
        return grid_adjacency(case["w"], case["h"], case["d"], case["length"], gen)
    return general_adjacency(case["n"], case["d"], case["s"], gen, _degrees(case))


def _batch_shapes(case):
    out = workloads.batch_shapes(case["count"], draw_seed=case["draw_seed"], n_lo=case["n_lo"], n_hi=case["n_hi"])
    for sh in out:
        if sh["grid"] and sh["symmetries"] == 4 and sh["degree"] % 4:
            sh["symmetries"] = 2
    return out


def _batch_spec(item):
    sh, seed = item
    gen, s = np.random.default_rng(seed), sh["symmetries"]
    if not sh["grid"]:
        return og.GraphSpec(general_adjacency(sh["nodes"], sh["degree"], s, gen), nodes=sh["nodes"], symmetries=s)
    w, h = sh["width"], sh["height"]
    return og.GraphSpec(grid_adjacency(w, h, sh["degree"], sh["length"], gen, s), grid=True, width=w, height=h,
                        symmetries=s)


def _batch_specs(case, seed):
    items = [(sh, [seed, i]) for i, sh in enumerate(_batch_shapes(case))]
    with ThreadPoolExecutor(8) as ex:
        return list(ex.map(_batch_spec, items))


def _serve_sizes(case):
    k = case["chains"]
    return [int(round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** (i / max(1, k - 1)))) for i in range(k)]


def _serve_graphs(case, seed):
    """Per chain: (GraphSpec, the move's deltas, the deltas that undo it)."""
    out = []
    for i, n in enumerate(_serve_sizes(case)):
        gen = np.random.default_rng([seed, i])
        adj = general_adjacency(n, case["d"], 1, gen)
        moved = adj.copy()
        r = og.Rng(int(gen.integers(1, 1 << 30))).mutate_general(n, case["d"], moved)
        move = og.two_opt_deltas(moved, r, n)
        undo = [(row, slot, int(adj[row, slot])) for row, slot, _ in move]
        out.append((og.GraphSpec(adj, nodes=n), moved, move, undo))
    return out


# --------------------------------------------------------------------------
# The calls.
# --------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("general", "grid"):
        adj, nd = _graph(case, seed), _degrees(case)
        if kind == "grid":
            og.init_aspl_grid(case["w"], case["h"], case["d"], nd)
        elif case["s"] > 1:
            og.init_aspl_general_s(case["n"], case["d"], nd, case["s"])
        else:
            og.init_aspl_general(case["n"], case["d"], nd)
        return dict(kind=kind, adj=adj)
    if kind == "batch":
        return dict(kind=kind, batch=og.Batch(_batch_specs(case, seed)))
    if kind == "serve":
        server = og.Server(max_nodes=case["n_hi"], memory_mb=256)
        chains = [(server.register(spec), move, undo) for spec, _, move, undo in _serve_graphs(case, seed)]
        return dict(kind=kind, server=server, chains=chains, moved=False)
    gen = np.random.default_rng(seed)
    chains = [og.Chain(general_adjacency(case["n"], case["d"], 1, gen), nodes=case["n"],
                       seed=int(gen.integers(1, 1 << 30)), max_temp=100.0, min_temp=0.2, ncalcs=10000)
              for _ in range(case["chains"])]
    return dict(kind=kind, anneal=og.Anneal(chains), count=len(chains), steps=case["steps"])


def _columns(results):
    d, s, a = zip(*results)
    return dict(diameter=np.array(d, dtype=np.int64), sum=np.array(s, dtype=np.int64),
                aspl=np.array(a, dtype=np.float64))


def run(state):
    kind = state["kind"]
    if kind in ("general", "grid"):
        d, s, a = og.set_aspl(state["adj"])
        return dict(diameter=d, sum=s, aspl=a)
    if kind == "batch":
        return _columns(state["batch"].run())
    if kind == "serve":
        server, moved = state["server"], state["moved"]
        state["moved"] = not moved                       # a move, then its rejection, and so on
        ids = [server.submit(h, undo if moved else move) for h, move, undo in state["chains"]]
        return _columns([server.wait(r)[:3] for r in ids])
    state["anneal"].run(state["steps"])
    st = [state["anneal"].state(k, graphs=True) for k in range(state["count"])]
    keys = ("steps", "accepted", "status", "diameter", "sum", "best_diameter", "best_sum")
    return dict(counts=np.array([[x[k] for k in keys] for x in st], dtype=np.int64),
                values=np.array([[x["aspl"], x["best_aspl"], x["temp"]] for x in st]),
                adjacency=np.stack([x["adjacency"] for x in st]),
                best_adjacency=np.stack([x["best_adjacency"] for x in st]))


# --------------------------------------------------------------------------
# Work and exact values.
# --------------------------------------------------------------------------

def _low_levels(n, d, reach=0, w=0, h=0):
    """Levels that no graph of the shape does without: the Moore bound, or
    corner to corner of a grid at `reach` per hop."""
    ball, shell, k = 1, d, 0
    while ball < n:
        ball, shell, k = ball + shell, shell * max(1, d - 1), k + 1
    return max(k, -(-(w + h - 2) // reach)) if reach else k


def _graph_work(n, d, s, levels):
    """(bytes of the adjacency and the results, 32-bit ORs of the levels)."""
    return 4.0 * (n // s) * d + 20, float(levels) * n * d * -(-(n // s) // 32)


def work(case):
    kind = case["kind"]
    if kind == "general":
        b, f = _graph_work(case["n"], case["d"], case["s"], _low_levels(case["n"], case["d"]))
    elif kind == "grid":
        n, lv = case["w"] * case["h"], _low_levels(case["w"] * case["h"], case["d"], case["length"], case["w"], case["h"])
        b, f = _graph_work(n, case["d"], 1, lv)
    elif kind == "batch":
        b = f = 0.0
        for sh in _batch_shapes(case):
            lv = _low_levels(sh["nodes"], sh["degree"], sh.get("length", 0), sh.get("width", 0), sh.get("height", 0))
            x, y = _graph_work(sh["nodes"], sh["degree"], sh["symmetries"], lv)
            b, f = b + x, f + y
    elif kind == "serve":
        b = 68.0 * case["chains"]                        # four updated slots in, one result out
        f = sum(_graph_work(n, case["d"], 1, _low_levels(n, case["d"]))[1] for n in _serve_sizes(case))
    else:
        b, f = _graph_work(case["n"], case["d"], 1, _low_levels(case["n"], case["d"]))
        b, f = 2 * b * case["chains"], f * case["chains"] * case["steps"]
    return {"bytes": b, "flops": f}


def _full_table(adj, n, s, nd, grid, w, h):
    """Neighbours of all n vertices (int64[n][d]; the vertex itself where it has none) and the base vertices."""
    base, d = adj.shape
    deg = np.full(base, d) if nd is None else nd
    a = np.where(np.arange(d)[None, :] < deg[:, None], adj, -1).astype(np.int64)
    full = np.empty((n, d), dtype=np.int64)
    if grid and s > 1:
        v = _base_vertices(w, h, s)
        for t in range(s):
            row = _rotate(v, w, h, s, t)
            full[row] = np.where(a < 0, row[:, None], _rotate(np.maximum(a, 0), w, h, s, t))
        return full, v
    for t in range(s):
        v = np.arange(base) + t * base
        full[v] = np.where(a < 0, v[:, None], (np.maximum(a, 0) + t * base) % n)
    return full, np.arange(base)


def _popcount(x):
    x = x - ((x >> 1) & 0x5555555555555555)
    x = (x & 0x3333333333333333) + ((x >> 2) & 0x3333333333333333)
    x = (x + (x >> 4)) & 0x0f0f0f0f0f0f0f0f
    return int(((x * 0x0101010101010101) >> 56).sum())


def _exact_aspl(adj, n, s, nd=None, grid=False, w=0, h=0):
    """(diameter, sum, ASPL) by breadth-first search over 64-bit words of sources."""
    full, sources = _full_table(adj, n, s, nd, grid, w, h)
    nbr = torch.from_numpy(full).cuda()
    total, diameter = 0, 0
    for c in range(0, len(sources), 4096):
        src = torch.from_numpy(sources[c:c + 4096]).cuda()
        i = torch.arange(len(src), device="cuda")
        bits = torch.zeros((n, -(-len(src) // 64)), dtype=torch.int64, device="cuda")
        bits[src, i // 64] = torch.ones_like(i) << (i % 64)
        full_count, count, level = n * len(src), len(src), 0
        while count < full_count:
            total += (full_count - count) * s
            new = bits.clone()
            for j in range(nbr.shape[1]):
                new |= bits[nbr[:, j]]
            bits, level, last = new, level + 1, count
            count = _popcount(bits)
            if count == last:
                return 2**31 - 1, 2**63 - 1, float(np.finfo(np.float64).max)
        diameter = max(diameter, level)
    return diameter, total // 2, total / ((float(n) - 1) * n)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("general", "grid"):
        adj, nd = _graph(case, seed), _degrees(case)
        if kind == "grid":
            r = _exact_aspl(adj, case["w"] * case["h"], 1, nd, True, case["w"], case["h"])
        else:
            r = _exact_aspl(adj, case["n"], case["s"], nd)
        return dict(diameter=r[0], sum=r[1], aspl=r[2])
    if kind == "batch":
        return _columns([_exact_aspl(g.adjacency, g.nodes, g.symmetries, None, g.grid, g.width, g.height)
                         for g in _batch_specs(case, seed)])
    if kind == "serve":
        return _columns([_exact_aspl(moved, g.nodes, 1) for g, moved, _, _ in _serve_graphs(case, seed)])
    return None                                          # a chain's decisions follow from all its results
