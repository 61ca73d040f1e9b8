"""The closure engine's work as a user's program has it done, case by case.

Every case goes through the public entry points: a kept context (`grg.Context`)
that loads graph after graph and closes them, a batch context that closes many
graphs together (`grg.Batch`), an out-of-core set (`grg.Partitioned`), the
allocation-free call (`grg_closure_noalloc`), and the compressed edge stream in
both directions (`grg_export_csr5`, `grg_load_csr5`).

The graphs are the generator's (`grg_gen.py`) families -- dataflow, block-structured
dataflow, block-confined alias, points-to -- drawn here with torch, so that an
8M-edge graph takes milliseconds to make.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "graspan-g_gb300"))
import grg  # noqa: E402
import grg_gen as G  # noqa: E402

RULES = {"dataflow": G.DATAFLOW_RULES, "blocks": G.DATAFLOW_RULES, "alias": G.ALIAS_RULES, "pointsto": G.POINTSTO_RULES}
GRAMMARS = [(G.DATAFLOW_RULES, G.grammar_labels(G.DATAFLOW_RULES)), (G.ALIAS_RULES, G.grammar_labels(G.ALIAS_RULES))]
EXITS, ENTRIES, CALLS = 10, 10, 5          # block-structured dataflow: see grg_gen.dataflow_blocks
DENSE_MAX = 12_000                         # vertices up to which exact() closes a graph as dense matrices


def listed():
    return [
        # One small program's points-to analysis: the shortest call there is, all launches and
        # waits. Every closure case reads its label counts, hash and degree table.
        {"name": "pointsto_600", "path": "closure", "graph": "pointsto", "vars": 600, "edges": 1800, "block": 0,
         "filter": 0},
        # A caller that may not allocate device memory closes one file's alias graph (three
        # procedures) in the static scratch array.
        {"name": "noalloc_alias_3k", "path": "noalloc", "graph": "alias", "vars": 3_000, "edges": 12_000,
         "block": 1000, "filter": 0},
        # The plain dataflow closure: 10,000 vertices, 30,000 edges, no blocks, filter 0. Every
        # row reaches nearly every vertex, in some 50 rounds.
        {"name": "dataflow_10k", "path": "closure", "graph": "dataflow", "vars": 10_000, "edges": 30_000, "block": 0,
         "filter": 0},
        # A library's alias analysis: an odd number of vertices, a ragged last procedure.
        {"name": "alias_37k", "path": "closure", "graph": "alias", "vars": 37_123, "edges": 148_492, "block": 1000,
         "filter": 0},
        # A mid-sized program's dataflow closure under filter 1, odd block size.
        {"name": "blocks_97k", "path": "closure", "graph": "blocks", "vars": 97_097, "edges": 291_291, "block": 1001,
         "filter": 1},
        # The benchmark's graph: 2,000 procedures of 1,000 vertices, 6M edges and their seeds.
        {"name": "blocks_2m", "path": "closure", "graph": "blocks", "vars": 2_000_000, "edges": 6_000_000,
         "block": 1000, "filter": 1},
        # The alias configuration: 1M vertices, 4M base edges and their inverses.
        {"name": "alias_1m", "path": "closure", "graph": "alias", "vars": 1_000_000, "edges": 4_000_000, "block": 1000,
         "filter": 0},
        # The largest in-core alias closure: half of the 8M-vertex configuration's graph at its
        # density (5 base edges a vertex).
        {"name": "alias_4m", "path": "closure", "graph": "alias", "vars": 4_000_000, "edges": 20_000_000,
         "block": 1000, "filter": 0},
        # A service's batch: jobs of uneven sizes, half dataflow and half alias, admitted from
        # host memory and closed together.
        {"name": "batch_24", "path": "batch", "graph": "mix", "jobs": 24, "vmin": 1_000, "vmax": 100_000,
         "density": 4.0, "vars": 24 * 21_500, "edges": 24 * 86_000, "block": 1000, "filter": 0},
        # The same closures out of core: partitions through host memory, with calls that cross
        # them, so pairs run.
        {"name": "parts_200k", "path": "parts", "graph": "alias", "vars": 200_000, "edges": 800_000, "block": 1000,
         "filter": 0, "parts": 8, "partner": 25},
        # Spilling a closed graph: the compressed stream into page-locked host memory.
        {"name": "stream_out_200k", "path": "out", "graph": "blocks", "vars": 200_000, "edges": 600_000,
         "block": 1000, "filter": 1},
        # Reading that spill back.
        {"name": "stream_in_200k", "path": "in", "graph": "blocks", "vars": 200_000, "edges": 600_000, "block": 1000,
         "filter": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges; sizes spread over their logarithm."""
    kind = rng.choice(["pointsto", "noalloc", "dataflow", "alias", "alias", "blocks", "blocks", "batch", "parts", "out",
                       "in"])
    if kind == "pointsto":
        v = _log(rng, 600, 2_000)
        return {"path": "closure", "graph": "pointsto", "vars": v, "edges": 3 * v, "block": 0, "filter": 0}
    if kind == "noalloc":
        v = _log(rng, 500, 3_000)
        return {"path": "noalloc", "graph": "alias", "vars": v, "edges": 4 * v, "block": rng.randint(200, 1000),
                "filter": 0}
    if kind == "dataflow":
        v = _log(rng, 500, 10_000)
        return {"path": "closure", "graph": "dataflow", "vars": v, "edges": 3 * v, "block": 0, "filter": 0}
    if kind == "alias":
        v = _log(rng, 5_000, 1_500_000)
        return {"path": "closure", "graph": "alias", "vars": v, "edges": int(v * rng.uniform(3, 5)),
                "block": rng.randint(500, 1000), "filter": 0}
    if kind == "blocks":
        b = rng.randint(500, 1001)
        nb = _log(rng, 6, 2_000)
        return {"path": "closure", "graph": "blocks", "vars": nb * b, "edges": 3 * nb * b, "block": b,
                "filter": rng.choice([0, 1])}
    if kind == "batch":
        jobs, top = rng.randint(3, 24), _log(rng, 10_000, 100_000)
        mean = int((top - 1_000) / math.log(top / 1_000))
        return {"path": "batch", "graph": "mix", "jobs": jobs, "vmin": 1_000, "vmax": top, "density": 4.0,
                "vars": jobs * mean, "edges": 4 * jobs * mean, "block": 1000, "filter": 0}
    if kind == "parts":
        v = _log(rng, 20_000, 200_000)
        return {"path": "parts", "graph": "alias", "vars": v, "edges": 4 * v, "block": 1000, "filter": 0,
                "parts": rng.randint(2, 8), "partner": max(1, v // 8000)}
    b = rng.randint(500, 1001)
    nb = _log(rng, 10, 200)
    return {"path": kind, "graph": "blocks", "vars": nb * b, "edges": 3 * nb * b, "block": b, "filter": 1}


# ---------------------------------------------------------------- graphs

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Rng:
    def __init__(self, seed):
        self.dev = _device()
        self.g = torch.Generator(device=self.dev).manual_seed(int(seed))

    def unit(self, n):
        return torch.rand(n, generator=self.g, device=self.dev, dtype=torch.float64)

    def ints(self, lo, hi, n):                     # lo <= x < hi
        return torch.randint(lo, hi, (n,), generator=self.g, device=self.dev, dtype=torch.int64)


def _zipf_sources(r, vertices, s, cap, total):
    """`total` source vertices: every vertex once, the rest by Zipf(s) out-degrees capped at `cap`."""
    n = vertices.numel()
    k = torch.arange(1, 1 << 16, device=r.dev, dtype=torch.float64).pow(-s)
    cdf = torch.cumsum(k, 0) / k.sum()
    extra = torch.clamp(torch.searchsorted(cdf, r.unit(n)) + 1, max=cap) - 1
    src = torch.repeat_interleave(vertices, extra)
    need = max(total - n, 0)
    if src.numel() > need:
        src = src[torch.randperm(src.numel(), generator=r.g, device=r.dev)[:need]]
    elif src.numel() < need:
        src = torch.cat([src, vertices[r.ints(0, n, need - src.numel())]])
    return torch.cat([vertices, src])


def _near(r, src, lo, hi, window):
    """Destinations within +-window of the source with probability 0.8, else uniform, in [lo, hi]."""
    m = src.numel()
    d_loc = torch.minimum(torch.maximum(src + r.ints(-window, window + 1, m), lo), hi)
    d_uni = lo + (r.unit(m) * (hi - lo + 1).double()).long()
    return torch.where(r.unit(m) < 0.8, d_loc, d_uni)


def _edges(case, seed):
    """(vars, src, dst, lab) as int64 tensors, sorted by source, without repeats."""
    r = _Rng(seed)
    V, E, block, kind = case["vars"], case["edges"], case["block"], case["graph"]
    labels = G.grammar_labels(RULES[kind])
    ids = {x: i + 1 for i, x in enumerate(labels)}
    every = torch.arange(V, device=r.dev)
    if kind == "blocks":
        nb = V // block
        V = nb * block
        every = every[:V]
        body = every[every % block < block - EXITS]
        exits = every[every % block >= block - EXITS]
        n_cross = min(E - int(round(E * 0.85)), exits.numel() * CALLS * ENTRIES)
        src = _zipf_sources(r, body, 2.0, 64, E - n_cross)
        lo = src // block * block
        dst = _near(r, src, lo, lo + (block - EXITS - 1), 256)
        xs = _zipf_sources(r, exits, 2.0, CALLS * ENTRIES, n_cross)
        xd = (xs // block + 1 + r.ints(0, CALLS, xs.numel())) % nb * block + r.ints(0, ENTRIES, xs.numel())
        src, dst = torch.cat([src, xs]), torch.cat([dst, xd])
        lab = torch.full_like(src, ids["e"])
        if case["filter"]:                          # filter 1 never applies N ::= e: seeds stand in for it
            src, dst = torch.cat([src, src]), torch.cat([dst, dst])
            lab = torch.cat([lab, torch.full_like(lab, ids["N"])])
    else:
        s, cap, window, frac = {"dataflow": (2.0, 64, 256, 0.0), "pointsto": (2.0, 64, 64, 0.4),
                                "alias": (1.8, 256, 256, 0.6)}[kind]
        src = _zipf_sources(r, every, s, cap, E)
        lo = src // block * block if block else torch.zeros_like(src)
        hi = torch.clamp(lo + block - 1, max=V - 1) if block else torch.full_like(src, V - 1)
        dst = _near(r, src, lo, hi, window)
        if case.get("partner"):                     # 2% of the calls go to the partner block
            p, nb = case["partner"], -(-V // block)
            b = src // block
            pb = torch.where((b // p) % 2 == 0, b + p, b - p)
            over = (r.unit(src.numel()) < 0.02) & (pb >= 0) & (pb < nb)
            dst = torch.where(over, torch.clamp(pb * block + (dst - lo), max=V - 1), dst)
        if kind == "dataflow":
            lab = torch.full_like(src, ids["e"])
        else:
            bar = (lambda x: x + "_bar") if kind == "alias" else (lambda x: "-" + x)
            is_a = r.unit(src.numel()) < frac
            lab = torch.where(is_a, ids["a"], ids["d"])
            inv = torch.where(is_a, ids[bar("a")], ids[bar("d")])
            src, dst, lab = torch.cat([src, dst]), torch.cat([dst, src]), torch.cat([lab, inv])
    key = torch.unique((src * V + dst) * 64 + lab)
    return V, key // 64 // V, key // 64 % V, key % 64


def _jobs(case, seed):
    """The batch's graphs: sizes log-uniform in [vmin, vmax] (the same for every seed), dataflow and
    alias in turn, host arrays."""
    out = []
    n = case["jobs"]
    for j in range(n):
        v = int(case["vmin"] * (case["vmax"] / case["vmin"]) ** ((j * 7 % n + 0.5) / n))
        kind = "blocks" if j % 2 == 0 else "alias"
        e = int(case["density"] * v)
        sub = {"graph": kind, "vars": max(v, case["block"]), "edges": e if kind == "blocks" else e // 2,
               "block": case["block"], "filter": 0}
        V, s, d, l = _edges(sub, seed * 1009 + j)
        out.append((j % 2, V, _host(s, np.uint32), _host(d, np.uint32), _host(l, np.uint8)))
    return out


def _host(t, dtype):
    return np.ascontiguousarray(t.cpu().numpy().astype(dtype))


def _rule_ids(kind):
    rules = RULES[kind]
    labels = G.grammar_labels(rules)
    ids = np.zeros((len(rules), 3), dtype=np.int32)
    for i, rule in enumerate(rules):
        for j, x in enumerate(rule):
            ids[i, j] = labels.index(x) + 1
    return ids, len(labels)


# ---------------------------------------------------------------- prepare and run

def _context(kind):
    ctx = grg.Context(torch.cuda.current_device())
    ids, n = _rule_ids(kind)
    ctx.transfer_rules(ids, n)
    ctx.allocate_pool(0)
    return ctx


def prepare(case, seed):
    path = case["path"]
    st = {"case": case}
    if path == "batch":
        st["jobs"] = _jobs(case, seed)
        st["vars"] = sum(j[1] for j in st["jobs"])
        st["ctx"] = grg.Context(torch.cuda.current_device())
        st["ctx"].allocate_pool(0)
        return st
    V, s, d, l = _edges(case, seed)
    st["vars"] = V
    if path == "parts":
        st["edges"] = (_host(s, np.uint32), _host(d, np.uint32), _host(l, np.uint8))
        st["ctx"] = _context(case["graph"])
        return st
    st["src"], st["dst"], st["lab"] = s.to(torch.int32), d.to(torch.int32), l.to(torch.uint8)
    torch.cuda.synchronize()
    if path == "noalloc":
        ids, n = _rule_ids(case["graph"])
        st["rules"], st["labels"] = np.ascontiguousarray(ids.reshape(-1)), n
        st["lib"] = grg.load_library()
        st["counts"] = torch.zeros(n, dtype=torch.int64, device="cuda")
        st["hash"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        return st
    st["ctx"] = _context(case["graph"])
    st["degrees"] = torch.zeros((6, V), dtype=torch.int32, pin_memory=True)
    if path == "closure":
        return st
    # a closed graph and the page-locked buffers its stream goes to (and comes from), with room
    # for a block's destinations in every row
    ctx = st["ctx"]
    _load(st)
    ctx.closure(case["filter"])
    st["room"] = V * case["block"]
    st["stream"] = torch.zeros(5 * st["room"], dtype=torch.uint8, pin_memory=True)
    st["degree"] = torch.empty(V, dtype=torch.int32, pin_memory=True)
    if path == "in":
        st["n"] = _export(st)
    return st


def _load(st):
    st["ctx"].load_edges_device(st["vars"], st["src"].numel(), st["src"].data_ptr(), st["dst"].data_ptr(),
                                st["lab"].data_ptr())


def _export(st):
    ctx, n = st["ctx"], ctypes.c_uint64()
    ctx._check(ctx._L.grg_export_csr5(ctx._h, 0, st["vars"], st["room"], ctypes.c_void_p(st["stream"].data_ptr()),
                                      ctypes.c_void_p(st["degree"].data_ptr()), ctypes.byref(n)), "export_csr5")
    return n.value


def _read(st):
    """What a caller reads of a loaded or closed graph: counts by label, the edge set's hash, and the
    edges and elements of every vertex."""
    ctx = st["ctx"]
    out = {"counts": _i64(ctx.label_counts()), "hash": _i64(ctx.set_hash())}
    ctx._check(ctx._L.grg_get_degree(ctx._h, 0, st["vars"] - 1, ctypes.c_void_p(st["degrees"].data_ptr())), "get_degree")
    out["edges"], out["elements"] = st["degrees"][0], st["degrees"][3]
    return out


def _i64(x):
    """Unsigned 64-bit results as int64 arrays of the same bits."""
    return np.atleast_1d(np.asarray(x, dtype=np.uint64)).view(np.int64)


def run(st):
    path, case = st["case"]["path"], st["case"]
    if path == "closure":
        # load a graph that is on the device, close it, read the result
        ctx = st["ctx"]
        _load(st)
        ctx.closure(case["filter"])
        return _read(st)
    if path == "noalloc":
        L, p = st["lib"], ctypes.c_void_p
        rounds = ctypes.c_uint64()
        r = L.grg_closure_noalloc(st["src"].device.index or 0, p(torch.cuda.current_stream().cuda_stream),
                                  len(st["rules"]) // 3, p(st["rules"].ctypes.data), st["labels"], case["filter"],
                                  st["vars"], st["src"].numel(), p(st["src"].data_ptr()), p(st["dst"].data_ptr()),
                                  p(st["lab"].data_ptr()), p(st["counts"].data_ptr()), p(st["hash"].data_ptr()),
                                  ctypes.byref(rounds))
        if r != grg.OK:
            raise grg.GrgError(r, grg.error_string(r))
        return {"counts": st["counts"], "hash": st["hash"]}
    if path == "batch":
        batch = grg.Batch(st["ctx"], st["vars"], len(st["jobs"]), GRAMMARS, 0)
        base = 0
        for j, (g, V, s, d, l) in enumerate(st["jobs"]):
            batch.admit(j, base, g, V, s, d, l)
            base += V
        batch.step(0)
        counts, hashes = [], []
        for j, job in enumerate(st["jobs"]):
            c, h = batch.result(j, job[0])
            counts.append(_i64(c))
            hashes.append(h)
        return {"counts": np.concatenate(counts), "hash": _i64(np.array(hashes, dtype=np.uint64))}
    if path == "parts":
        part = grg.Partitioned(st["ctx"], st["vars"], case["parts"])
        part.load_edges(*st["edges"])
        part.run(case["filter"])
        counts, h = part.label_counts()
        part.close()
        return {"counts": _i64(counts), "hash": _i64(h)}
    if path == "out":
        _export(st)
        return {"stream": st["stream"], "degree": st["degree"]}
    ctx = st["ctx"]
    ctx._check(ctx._L.grg_load_csr5(ctx._h, st["vars"], 0, st["vars"], ctypes.c_void_p(st["degree"].data_ptr()), st["n"],
                                    ctypes.c_void_p(st["stream"].data_ptr()), 0), "load_csr5")
    return _read(st)


# ---------------------------------------------------------------- work and the exact results

def _closure_size(case):
    """(closure edges, 192-id elements) of a case, about: a dataflow row reaches every vertex, a
    block-structured one two thirds of a block, an alias row has about 2.4 blocks of destinations
    over its derived labels."""
    V, block, kind = case["vars"], case["block"], case["graph"]
    if kind == "pointsto":
        return V * V * 555 // 100, 9 * V * (V // 192 + 1)
    if kind == "dataflow":
        return V * V * 93 // 100, V * (V // 192 + 1)
    width = block // 192 + 1
    if kind == "blocks":
        return V * block * 66 // 100, V * width
    if kind == "alias":
        return V * block * 237 // 100, 3 * V * width
    return V * block * 150 // 100, 2 * V * width


def work(case):
    """Bytes of a pass: each input edge (9 bytes) and each stored 32-byte element once; for the
    stream, its 5 bytes an edge, the row lengths and the elements once. A closure is a union of
    sets: no floating-point operations."""
    edges, elems = _closure_size(case)
    V, E = case["vars"], case["edges"]
    if case["graph"] in ("alias", "pointsto") or (case["graph"] == "blocks" and case["filter"]):
        E *= 2                                       # inverses, or seeds
    if case["path"] in ("out", "in"):
        return {"bytes": 5 * edges + 4 * V + 32 * elems, "flops": 0}
    return {"bytes": 9 * E + 32 * elems, "flops": 0}


def _mix64(x):
    """splitmix64 on int64 tensors (logical shifts)."""
    def shr(v, n):
        return (v >> n) & ((1 << (64 - n)) - 1)

    x = x + (0x9E3779B97F4A7C15 - (1 << 64))
    x = (x ^ shr(x, 30)) * (0xBF58476D1CE4E5B9 - (1 << 64))
    x = (x ^ shr(x, 27)) * (0x94D049BB133111EB - (1 << 64))
    return x ^ shr(x, 31)


def _dense(kind, V, s, d, l, filter_flag):
    """The closure as one 0/1 matrix a label, iterated to its fixpoint."""
    ids, n = _rule_ids(kind)
    M = [torch.zeros(V, V, device=s.device) for _ in range(n + 1)]
    for x in range(1, n + 1):
        at = l == x
        M[x][s[at], d[at]] = 1.0
    for A, B, _ in ids:
        if not B:
            M[A].fill_diagonal_(1.0)
    before = -1
    while True:
        now = sum(int(m.sum(dtype=torch.float64)) for m in M[1:])
        if now == before:
            return M
        before = now
        for A, B, C in ids:
            if C:
                M[A] = torch.maximum(M[A], (M[B] @ M[C] > 0).float())
            elif B and not filter_flag:
                M[A] = torch.maximum(M[A], M[B])


def _dense_results(kind, V, s, d, l, filter_flag):
    M = _dense(kind, V, s, d, l, filter_flag)
    counts, h = [], torch.zeros((), dtype=torch.int64, device=s.device)
    for x, m in enumerate(M[1:], 1):
        counts.append(int(m.sum(dtype=torch.float64)))
        e = m.nonzero()
        salt = (x * 0x9E3779B97F4A7C15) % (1 << 64)
        salt = salt - (1 << 64) if salt >> 63 else salt
        h = h + _mix64(_mix64((e[:, 0] << 32) | e[:, 1]) ^ salt).sum()
    out = {"counts": np.array(counts, dtype=np.int64), "hash": h.reshape(1).cpu().numpy()}
    out["edges"] = sum(m.sum(1, dtype=torch.float64) for m in M[1:]).to(torch.int32).cpu().numpy()
    pad = -V % 192
    units = [torch.nn.functional.pad(m, (0, pad)).reshape(V, -1, 192).amax(2).sum(1) for m in M[1:]]
    out["elements"] = sum(units).to(torch.int32).cpu().numpy()
    return out, M


def _dense_stream(M):
    """The compressed stream of the closed matrices: 5 bytes an edge, by row, label, destination."""
    e = torch.stack(M[1:], 1).nonzero()
    b = torch.stack([(e[:, 2] >> (8 * i)) & 255 for i in range(4)] + [e[:, 1] + 1], 1)
    return b.to(torch.uint8).reshape(-1)


def exact(case, seed):
    path = case["path"]
    if path == "batch":
        counts, hashes = [], []
        for g, V, s, d, l in _jobs(case, seed):
            if V > DENSE_MAX:
                return None
            kind = ("blocks", "alias")[g]
            e = [torch.from_numpy(x.astype(np.int64)).to(_device()) for x in (s, d, l)]
            r, _ = _dense_results(kind, V, *e, 0)
            counts.append(r["counts"])
            hashes.append(r["hash"])
        return {"counts": np.concatenate(counts), "hash": np.concatenate(hashes)}
    if case["vars"] > DENSE_MAX:
        return None
    V, s, d, l = _edges(case, seed)
    r, M = _dense_results(case["graph"], V, s, d, l, case["filter"])
    if path == "out":
        stream = torch.zeros(5 * V * case["block"], dtype=torch.uint8)
        b = _dense_stream(M).cpu()
        stream[:b.numel()] = b
        return {"stream": stream, "degree": r["edges"]}
    return {k: r[k] for k in ("counts", "hash")} if path == "noalloc" else r
