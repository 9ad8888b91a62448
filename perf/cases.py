"""The measured workloads of the miner: what a user's program has it do, through its public entry points.

Databases come from the package's seeded generator (its configurations 1-5) or, for graphs beyond 64 vertices, from
seeded arrays of the shape the tests use.  Pattern lists are taken in the library's bulk form (gs_mine_collect,
gs_server_poll), as numpy arrays: pattern i is dfs[offset[i]:offset[i + 1]] with support[i].
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

import gpu_graph_mining_gb300 as gs


def listed():
    return [
        # the reference's own test database shape (340 molecules): a short interactive call, launches and host waits
        {"name": "chem340_s20pct", "kind": "mine", "config": 1, "scale": 1.0, "frac": 0.20},
        # the same database mined deep: thousands of patterns, few embeddings each
        {"name": "chem340_s5pct", "kind": "mine", "config": 1, "scale": 1.0, "frac": 0.05},
        # the plain one-pattern-at-a-time form (wave_nodes = 1), as the reference drives its kernels
        {"name": "chem340_plain", "kind": "mine", "config": 1, "scale": 1.0, "frac": 0.20, "wave_nodes": 1},
        # the generator-style database at its lowest support: the ordinary mining call
        {"name": "graphs100k_s1pct", "kind": "mine", "config": 2, "scale": 1.0, "frac": 0.01},
        # an odd-sized database with the pattern-size cap of a serving request
        {"name": "graphs23k_s2pct_e5", "kind": "mine", "config": 2, "scale": 0.23457, "frac": 0.02, "max_edges": 5},
        # a database whose adjacency (240 MB) is larger than L2, at half a percent: the largest call
        {"name": "graphs250k_s0.5pct", "kind": "mine", "config": 5, "scale": 0.25, "frac": 0.005},
        # the lists extension strategy
        {"name": "graphs50k_lists", "kind": "mine", "config": 2, "scale": 0.5, "frac": 0.01, "extension": "lists"},
        # from the reference's host arrays to all patterns: device ingest, then mining
        {"name": "graphs100k_arrays", "kind": "arrays", "config": 2, "scale": 1.0, "frac": 0.02},
        # many databases mined together
        {"name": "batch64", "kind": "batch", "count": 64, "scale": 0.2, "frac": 0.05},
        # a burst of requests on resident databases, mined with continuous batching
        {"name": "serve8x32", "kind": "serve", "count": 8, "scale": 0.2, "requests": 32},
        # graphs beyond 64 vertices: the general membership test
        {"name": "large_graphs_e5", "kind": "large", "graphs": 3001, "vmin": 60, "vmax": 130, "frac": 0.5, "max_edges": 5},
        # support counting as an operator on a caller's device buffers
        {"name": "support_4m", "kind": "support", "records": 4000003, "keys": 1000, "graphs": 30011},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["mine", "mine", "mine", "mine", "arrays", "batch", "serve", "large", "support"])
    if kind in ("mine", "arrays"):
        config = rng.choice([1, 2, 2, 5])
        c = {"kind": kind, "config": config}
        if config == 1:
            c["scale"] = round(_log(rng, 1.0, 20.0), 4)
            c["frac"] = round(_log(rng, 0.05, 0.34), 4)
        elif config == 2:
            c["scale"] = round(_log(rng, 0.02, 1.0), 4)
            c["frac"] = round(_log(rng, 0.01, 0.05), 4)
        else:
            c["scale"] = round(_log(rng, 0.01, 0.24), 4)
            c["frac"] = round(_log(rng, 0.005, 0.02), 4)
        if rng.random() < 0.3:
            c["max_edges"] = rng.randint(4, 8)
        if kind == "mine" and rng.random() < 0.2:
            c["extension"] = "lists"
        return c
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 64), "scale": round(_log(rng, 0.05, 0.2), 4),
                "frac": round(_log(rng, 0.05, 0.1), 4)}
    if kind == "serve":
        return {"kind": kind, "count": rng.randint(2, 8), "scale": round(_log(rng, 0.05, 0.2), 4),
                "requests": rng.randint(4, 48)}
    if kind == "large":
        return {"kind": kind, "graphs": int(_log(rng, 300, 3000)), "vmin": rng.randint(20, 66),
                "vmax": rng.randint(70, 200), "frac": round(rng.uniform(0.5, 0.8), 3), "max_edges": rng.randint(3, 5)}
    graphs = int(_log(rng, 100, 100000))
    return {"kind": kind, "records": int(_log(rng, 1000, 4000000)), "graphs": graphs,
            "keys": int(_log(rng, 1, (1 << 20) // ((graphs + 31) // 32)))}


# ------------------------------------------------------------------ preparation

def _minsup(db, frac):
    return max(2, int(round(frac * len(db))))


def _options(case):
    o = gs.MineOpts()
    gs.lib().gs_mine_opts_default(ctypes.byref(o))
    o.max_edges = case.get("max_edges", 0)
    o.wave_nodes = case.get("wave_nodes", o.wave_nodes)
    o.extension = {"rmpath": gs.EXTENSION_RMPATH, "lists": gs.EXTENSION_LISTS}[case.get("extension", "rmpath")]
    return o


def _cudabin(db):
    """The reference's flat cudabin arrays of a database, in host memory."""
    fd, path = tempfile.mkstemp(suffix=".cudabin")
    os.close(fd)
    try:
        db.write(path, "cudabin")
        raw = np.fromfile(path, dtype=np.int32)
    finally:
        os.remove(path)
    n, esz, maxv = (int(x) for x in raw[:3])
    cuts = np.cumsum([4, esz, esz, n * maxv, n * maxv + 1])
    e, el, vl, vo = (raw[a:b].copy() for a, b in zip(cuts[:-1], cuts[1:]))
    return n, maxv, e, el, vl, vo


def _large_arrays(case, seed):
    """Random connected graphs of vmin..vmax vertices (a random tree and nv / 8 chords), as cudabin arrays."""
    r = np.random.default_rng([seed, 7])
    n, maxv = case["graphs"], case["vmax"]
    nv = r.integers(case["vmin"], maxv + 1, n)
    g = np.repeat(np.arange(n), nv)
    first = np.repeat(np.cumsum(nv) - nv, nv)
    v = np.arange(g.size) - first
    tree = v > 0
    a, b, eg = (r.random(g.size) * v).astype(np.int64)[tree], v[tree], g[tree]
    cg = np.repeat(np.arange(n), nv // 8)
    ca, cb = ((r.random(cg.size) * nv[cg]).astype(np.int64) for _ in range(2))
    ok = ca != cb
    a, b, eg = (np.concatenate(x) for x in ((a, np.minimum(ca, cb)[ok]), (b, np.maximum(ca, cb)[ok]), (eg, cg[ok])))
    code = np.unique((eg * maxv + a) * maxv + b)
    eg, a, b = code // (maxv * maxv), code // maxv % maxv, code % maxv
    lab = r.integers(0, 2, code.size)
    src = np.concatenate((eg * maxv + a, eg * maxv + b))
    dst = np.concatenate((eg * maxv + b, eg * maxv + a))
    lab = np.concatenate((lab, lab))
    order = np.lexsort((dst, src))
    off = np.concatenate(([0], np.cumsum(np.bincount(src, minlength=n * maxv))))
    pad = np.arange(n * maxv) % maxv >= np.repeat(nv, maxv)
    off[:-1][pad] = -1
    vl = np.where(pad, -1, r.choice([0, 0, 1, 2], n * maxv))
    return n, maxv, dst[order], lab[order], vl, off


def prepare(case, seed):
    kind = case["kind"]
    if kind == "support":
        g = torch.Generator(device="cuda").manual_seed(seed)
        # extension records as they arrive: candidate keys with a skewed frequency, graph ids in any order
        u = torch.rand(case["records"], generator=g, device="cuda")
        keys = (u * u * case["keys"]).to(torch.int32).clamp_(max=case["keys"] - 1)
        gids = torch.randint(0, case["graphs"], (case["records"],), generator=g, device="cuda", dtype=torch.int32)
        return {"case": case, "keys": keys, "gids": gids,
                "out": torch.empty(case["keys"], dtype=torch.int32, device="cuda")}
    if kind in ("batch", "serve"):
        config = 3 if kind == "batch" else 4
        dbs = [gs.Database.generate(config, seed=1 + seed * 64 + i, scale=case["scale"]) for i in range(case["count"])]
        for d in dbs:
            d.upload()
        if kind == "batch":
            return {"case": case, "dbs": dbs, "minsups": [_minsup(d, case["frac"]) for d in dbs]}
        r = np.random.default_rng([seed, 3])
        server = gs.Server()
        ids = [server.add_db(d) for d in dbs]
        reqs = []
        for _ in range(case["requests"]):
            k = int(r.integers(0, len(dbs)))
            reqs.append((ids[k], _minsup(dbs[k], float(r.choice([0.01, 0.02, 0.05, 0.10]))), int(r.integers(4, 9))))
        return {"case": case, "server": server, "requests": reqs,
                "out": _buffers(1 << 18, 4000000)}
    if kind == "large":
        n, maxv, e, el, vl, vo = _large_arrays(case, seed)
        db = gs.Database.from_arrays(n, maxv, e, el, vl, vo)
        db.upload()
        return {"case": case, "db": db, "minsup": _minsup(db, case["frac"]), "opts": _options(case),
                "out": _buffers(1 << 17, 1 << 21)}
    db = gs.Database.generate(case["config"], seed=1 + seed, scale=case["scale"])
    state = {"case": case, "minsup": _minsup(db, case["frac"]), "opts": _options(case),
             "out": _buffers(1 << 17, 1 << 21)}
    if kind == "arrays":
        state["arrays"] = _cudabin(db)
        db.free()
    else:
        db.upload()
        state["db"] = db
    return state


# ------------------------------------------------------------------ one pass

def _buffers(patterns, ints):
    """A caller's result buffers: room for so many patterns and DFS-code values; what a result does not fill stays 0."""
    return {"count": np.zeros(2, np.int64), "offset": np.zeros(patterns + 1, np.int64),
            "support": np.zeros(patterns, np.int64), "dfs": np.zeros(ints, np.int32)}


def _append(p, out, at):
    """Copies a native pattern list behind the patterns and tuples that out holds; the native buffer is freed."""
    try:
        c = p.contents
        n, t = at
        if c.count:
            out["offset"][n:n + c.count + 1] = np.ctypeslib.as_array(c.offset, shape=(c.count + 1,))
            out["offset"][n:n + c.count + 1] += t
            out["support"][n:n + c.count] = np.ctypeslib.as_array(c.support, shape=(c.count,))
            out["dfs"][5 * t:5 * (t + c.n_tuples)] = np.ctypeslib.as_array(c.dfs, shape=(5 * c.n_tuples,))
        return n + c.count, t + c.n_tuples
    finally:
        gs.lib().gs_patterns_free(p)


def _ok(status):
    if status:
        raise gs.GSpanError(status, gs.lib().gs_last_error().decode(errors="replace"))


def _collect(db, state):
    p = ctypes.POINTER(gs.Patterns)()
    _ok(gs.lib().gs_mine_collect(db.handle, state["minsup"], ctypes.byref(state["opts"]), ctypes.byref(p), None))
    state["out"]["count"][:] = _append(p, state["out"], (0, 0))
    return state["out"]


def run(state):
    kind = state["case"]["kind"]
    if kind == "support":
        k = state["keys"]
        _ok(gs.lib().gs_support_count_noalloc(k.data_ptr(), state["gids"].data_ptr(), k.numel(), state["case"]["keys"],
                                              state["case"]["graphs"], state["out"].data_ptr(),
                                              torch.cuda.current_stream().cuda_stream))
        return state["out"]
    if kind == "batch":
        # counting form: patterns per call, no sink (a Python sink would be most of the time)
        _, st = gs.mine_batch(state["dbs"], state["minsups"], collect=False)
        return [st["patterns"], st["nodes"]]
    if kind == "serve":
        rids = [state["server"].submit(*q) for q in state["requests"]]
        at = (0, 0)
        for rid in rids:
            p = ctypes.POINTER(gs.Patterns)()
            _ok(gs.lib().gs_server_poll(state["server"]._h, rid, -1, None, ctypes.byref(p)))
            at = _append(p, state["out"], at)
        state["out"]["count"][:] = at
        return state["out"]
    if kind == "arrays":
        n, maxv, e, el, vl, vo = state["arrays"]
        db = gs.Database.from_arrays(n, maxv, e, el, vl, vo, device=True)
        try:
            return _collect(db, state)
        finally:
            db.free()
    return _collect(state["db"], state)


# ------------------------------------------------------------------ work and exact values

def work(case):
    """Each input read once: a database's packed adjacency (8 bytes an entry), offsets, labels and graph ids (12 bytes
    a vertex); host arrays 8 bytes an entry and 8 a vertex slot.  Outputs (thousands of patterns) are small beside it."""
    kind = case["kind"]
    if kind == "support":
        return {"bytes": 8.0 * case["records"] + 4.0 * case["keys"], "flops": 0.0}
    if kind == "large":
        nv = 0.5 * (case["vmin"] + case["vmax"]) * case["graphs"]
        return {"bytes": 8.0 * 2.25 * nv + 12.0 * nv, "flops": 0.0}
    if kind in ("batch", "serve"):
        lo, hi, edges = (1000.0, 50000.0, 25.0) if kind == "batch" else (10000.0, 200000.0, 30.0)
        graphs = case["count"] * case["scale"] * (hi - lo) / math.log(hi / lo)
        return {"bytes": graphs * edges * (8.0 * 2 + 12.0), "flops": 0.0}
    graphs, edges = {1: (340, 36.0), 2: (100000, 30.0), 5: (1000000, 40.0)}[case["config"]]
    b = graphs * case["scale"] * edges * (8.0 * 2 + 12.0)
    return {"bytes": 2 * b if kind == "arrays" else b, "flops": 0.0}


def exact(case, seed):
    if case["kind"] != "support":
        return None
    s = prepare(case, seed)
    pairs = torch.unique(s["keys"].long() * case["graphs"] + s["gids"].long())
    return torch.bincount(pairs // case["graphs"], minlength=case["keys"]).to(torch.int32)
