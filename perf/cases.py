"""The calls of this engine whose speed is watched, over the sizes they are used at.

A case is a dict: `kind` names the entry point, the other keys its sizes and
options.  `listed()` gives the fixed cases, `draw(rng)` further ones of the
same ranges; `prepare` builds a case's graph and inputs from a seed, `run`
makes one call, `work` states the bytes and operations a call cannot do
without, `exact` what floating outputs are in 64 bits.

Graphs are R-MAT (0.57, 0.19, 0.19, 0.05), edge factor 16, as in the benchmark
and the tests.  The kinds:

  walks     Graph.walk_device over walk records in HBM (raw walks, graphlet
            closure, trajectories), every rule, both layouts and both RNG modes
  pools     Graph.run_pools: 64-bit walk words in pinned host memory, counts back
  ppr       Graph.ppr: one query, a few plain ones, or a batch (msppr)
  blocked   Graph.run through the block loop, the graph in HBM or streamed
            from pinned host memory
  simrank   Graph.simrank_batch
  visits    Graph.expected_visits (FP64)
  serve     Server.submit / wait of a burst of queries
"""
from __future__ import annotations

import math

import numpy as np
import torch

import graphwalker_b200 as gw

EF = 16
A, B, C = 0.57, 0.19, 0.19
THRESHOLD = 322122544  # a 31-bit draw r continues when (float)r / RAND_MAX > 0.15
RULES = {"jump": gw.RULE_JUMP, "stop": gw.RULE_STOP, "prob": gw.RULE_PROB, "restart": gw.RULE_RESTART,
         "ppr": gw.RULE_PPR}
SINKS = {"count": gw.SINK_VERTEX_COUNT, "path": gw.SINK_PATH_RECORD, "closure": gw.SINK_CLOSURE_COUNT}


def listed() -> list[dict]:
    return [
        # A short call: one small walk set on a small graph (the smoke test's walk count).
        {"name": "raw_small", "kind": "walks", "scale": 14, "walks": 4099, "rule": "jump", "sink": "count", "L": 10,
         "rng": "philox", "layout": "records"},
        # The headline workload: one walk per vertex at scale 24.
        {"name": "raw_headline", "kind": "walks", "scale": 24, "walks": 1 << 24, "rule": "jump", "sink": "count",
         "L": 10, "rng": "philox", "layout": "records"},
        # A corpus of trajectories (what node embeddings and SimRank read), an odd number of them.
        {"name": "raw_paths", "kind": "walks", "scale": 22, "walks": 3000001, "rule": "restart", "sink": "path",
         "L": 11, "rng": "philox", "layout": "records"},
        # The host program's call: walk words in, counts out.
        {"name": "host_pools", "kind": "pools", "scale": 22, "walks": 1 << 22, "rule": "jump", "L": 10},
        # One query of the serving workload's mean budget, on its own.
        {"name": "ppr_one", "kind": "ppr", "scale": 22, "queries": 1, "budget": 300, "spread": False, "rule": "ppr",
         "L": 20, "batched": False},
        # Single-source PPR: 100,000 walks at scale 20.
        {"name": "ppr_single", "kind": "ppr", "scale": 20, "queries": 1, "budget": 100000, "spread": False,
         "rule": "ppr", "L": 20, "batched": True},
        # The msppr batch: 4096 queries, budgets 10^U(2, 5).
        {"name": "msppr", "kind": "ppr", "scale": 24, "queries": 4096, "budget": 100000, "spread": True,
         "rule": "ppr", "L": 20, "batched": True},
        # The block loop with the graph in HBM, one walk per vertex.
        {"name": "block_loop", "kind": "blocked", "scale": 22, "blocks": 32, "resident": True, "walks": 1 << 22,
         "rule": "jump", "L": 10},
        # The same out of core: 73 % of the blocks on the device.
        {"name": "out_of_core", "kind": "blocked", "scale": 22, "blocks": 32, "resident": False, "walks": 1 << 22,
         "rule": "jump", "L": 10},
        # SimRank queries with the reference app's walk count and length.
        {"name": "simrank", "kind": "simrank", "scale": 20, "pairs": 512, "R": 1000, "L": 11},
        # The accuracy reference of a PPR query.
        {"name": "visits", "kind": "visits", "scale": 20, "rule": "ppr", "L": 20},
        # A burst of queries at the server, Pareto budgets (mean about 300).
        {"name": "serve_burst", "kind": "serve", "scale": 22, "queries": 256, "rule": "ppr", "L": 20},
    ]


def _log(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["walks", "walks", "walks", "pools", "ppr", "ppr", "ppr", "blocked", "blocked", "simrank",
                       "visits", "serve"])
    if kind == "walks":
        scale, sink = rng.randint(12, 23), rng.choice(["count", "count", "path", "closure"])
        return {"kind": kind, "scale": scale, "walks": _log(rng, 1000, min(1 << scale, 1 << 22)),
                "rule": rng.choice(["jump", "stop", "restart", "ppr"] + (["prob"] if sink != "path" else [])),
                "sink": sink, "L": rng.randint(4, 20), "rng": rng.choice(["philox", "philox", "native"]),
                "layout": rng.choice(["records", "records", "csr"])}
    if kind == "pools":
        scale = rng.randint(16, 22)
        return {"kind": kind, "scale": scale, "walks": _log(rng, 20000, 1 << scale), "rule": rng.choice(["jump", "stop"]),
                "L": rng.randint(5, 16)}
    if kind == "ppr":
        batched = rng.random() < 0.75
        queries = _log(rng, 1, 2048) if batched else rng.randint(1, 8)
        spread = rng.random() < 0.5
        return {"kind": kind, "scale": rng.randint(16, 23), "queries": queries, "spread": spread,
                "budget": _log(rng, 100, min(100000, (50000000 if spread else 10000000) // queries)), "rule": rng.choice(["ppr", "ppr", "stop", "restart"]),
                "L": rng.randint(8, 20), "batched": batched}
    if kind == "blocked":
        scale = rng.randint(18, 22)
        return {"kind": kind, "scale": scale, "blocks": rng.randint(4, 48), "resident": rng.random() < 0.5,
                "walks": _log(rng, 10000, 1 << scale), "rule": rng.choice(["jump", "stop", "restart"]),
                "L": rng.randint(5, 12)}
    if kind == "simrank":
        return {"kind": kind, "scale": rng.randint(14, 20), "pairs": _log(rng, 1, 512), "R": _log(rng, 100, 1000),
                "L": rng.randint(5, 16)}
    if kind == "visits":
        return {"kind": kind, "scale": rng.randint(14, 20), "rule": rng.choice(["ppr", "stop", "restart", "jump"]),
                "L": rng.randint(6, 20)}
    return {"kind": kind, "scale": rng.randint(16, 22), "queries": _log(rng, 8, 256), "rule": rng.choice(["ppr", "stop"]),
            "L": rng.randint(8, 20)}


class State(dict):
    """A case's graph and inputs; the server and the graph are closed with it."""

    def __del__(self):
        for key in ("server", "graph"):
            if key in self:
                self[key].close()


def _params(case, seed: int, **more):
    return gw.params(RULES[case.get("rule", "restart")], more.pop("sink", gw.SINK_VERTEX_COUNT), case["L"], seed=seed,
                     **more)


def _kb(scale: int, nblocks: int) -> int:
    return -(-EF * (1 << scale) * 4 // nblocks // 1024)


def _rmat(case, seed: int, nblocks: int = 32) -> gw.Graph:
    return gw.Graph.rmat(case["scale"], EF, seed=seed, blocksize_kb=_kb(case["scale"], nblocks))


def _sources(g: gw.Graph, n: int, r) -> np.ndarray:
    """n vertices with out-edges."""
    rowptr, _ = g.export_csr()
    return r.choice(np.flatnonzero(np.diff(rowptr) > 0), n).astype(np.uint32)


def _budgets(case, r) -> np.ndarray:
    n = case["queries"]
    if not case["spread"]:
        return np.full(n, case["budget"], np.uint32)
    return np.round(10 ** r.uniform(2, math.log10(max(case["budget"], 101)), n)).astype(np.uint32)


def _csr(scale: int, seed: int):
    """An R-MAT graph by torch alone (rowptr, colidx on the GPU), ids permuted, self-loops dropped."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    nv, m = 1 << scale, EF << scale
    src = torch.zeros(m, dtype=torch.int64, device="cuda")
    dst = torch.zeros_like(src)
    for _ in range(scale):
        u = torch.rand(m, generator=gen, device="cuda")
        src = src * 2 + (u >= A + B)
        dst = dst * 2 + (((u >= A) & (u < A + B)) | (u >= A + B + C))
    perm = torch.randperm(nv, generator=gen, device="cuda")
    src, dst = perm[src], perm[dst]
    key = (src * nv + dst)[src != dst].sort().values
    rowptr = torch.zeros(nv + 1, dtype=torch.int64, device="cuda")
    rowptr[1:] = torch.bincount(key // nv, minlength=nv).cumsum(0)
    return rowptr, key % nv


def _open(rowptr, colidx, nblocks: int = 16) -> gw.Graph:
    rp = rowptr.cpu().numpy().astype(np.uint64)
    ci = colidx.to(torch.int32).cpu().numpy().view(np.uint32)
    return gw.Graph.from_csr(rp, ci, gw.compute_blocks(rp, max(1, len(ci) * 4 // nblocks // 1024)))


def _pairs(case, rowptr, seed: int):
    r = np.random.default_rng(seed)
    with_edges = torch.nonzero(rowptr[1:] > rowptr[:-1]).flatten().cpu().numpy()
    v = r.choice(with_edges, (2, case["pairs"])).astype(np.uint32)
    return v[0].copy(), v[1].copy()


def prepare(case, seed: int):
    kind, r = case["kind"], np.random.default_rng(seed)
    s = State(case=case)
    if kind == "walks":
        g = s["graph"] = _rmat(case, seed)
        g.set_edge_records(gw.EDGE_RECORDS_OFF if case["layout"] == "csr" else gw.EDGE_RECORDS_ON)
        n, nv, L = case["walks"], g.nv, case["L"]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        cur = (torch.arange(n, device="cuda") if n == nv else
               torch.randint(0, nv, (n,), generator=gen, device="cuda"))
        rec = torch.stack([cur, torch.arange(n, device="cuda"), cur, torch.zeros_like(cur)], 1)
        s["walks"] = rec.to(torch.int32).contiguous()
        s["params"] = _params(case, seed, sink=SINKS[case["sink"]], rng=gw.RNG_NATIVE if case["rng"] == "native"
                              else gw.RNG_PHILOX, path_stride=L if case["sink"] == "path" else 0)
        if case["sink"] == "count":
            s["out"] = torch.zeros(nv, dtype=torch.int32, device="cuda")
        elif case["sink"] == "closure":
            s["out"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        else:
            s["out"] = torch.zeros((n, L), dtype=torch.int32, device="cuda")
            s["lens"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    elif kind == "pools":
        g = s["graph"] = _rmat(case, seed)
        n, nv = case["walks"], g.nv
        cur = np.arange(nv) if n == nv else np.sort(r.integers(0, nv, n))
        blk = np.searchsorted(g.blocks[1:], cur, side="right")
        words = gw.encode(cur, cur - g.blocks[blk].astype(np.int64), 0)
        offs = np.r_[0, np.cumsum(np.bincount(blk, minlength=g.nblocks))].astype(np.int64)
        s["words"] = torch.from_numpy(words.view(np.int64)).pin_memory()
        s["offsets"] = torch.from_numpy(offs).pin_memory()
        # one walk per vertex is keyed on its source; walks of any other set carry ids
        s["ids"] = None if n == nv else torch.arange(n, dtype=torch.int32).pin_memory()
        s["out"] = torch.zeros(nv, dtype=torch.int32).pin_memory()
        s["params"] = _params(case, seed)
    elif kind == "ppr":
        g = s["graph"] = _rmat(case, seed)
        s["sources"], s["budgets"] = _sources(g, case["queries"], r), _budgets(case, r)
        s["params"] = _params(case, seed)
    elif kind == "blocked":
        g = s["graph"] = _rmat(case, seed, case["blocks"])
        if not case["resident"]:
            g.set_residency(gw.STREAM_PINNED, max(2, g.nblocks * 73 // 100))
        n = case["walks"]
        cur = np.arange(n, dtype=np.uint32) if n == g.nv else np.sort(r.integers(0, g.nv, n).astype(np.uint32))
        g.add_walks_at(cur, ids=np.arange(n, dtype=np.uint32))
        s["params"] = _params(case, seed, mode=gw.MODE_BLOCKED)
    elif kind == "simrank":
        rowptr, colidx = _csr(case["scale"], seed)
        s["graph"] = _open(rowptr, colidx)
        s["a"], s["b"] = _pairs(case, rowptr, seed)
        s["seed"] = seed
    elif kind == "visits":
        rowptr, colidx = _csr(case["scale"], seed)
        s["graph"] = _open(rowptr, colidx)
        s["source"] = int(torch.argmax(rowptr[1:] - rowptr[:-1]))
        s["params"] = _params(case, seed)
    else:
        g = s["graph"] = _rmat(case, seed)
        s["sources"] = _sources(g, case["queries"], r)
        s["budgets"] = np.clip(100 * (1 + r.pareto(1.5, case["queries"])), 100, 100000).astype(np.uint32)
        s["server"] = g.serve(_params(case, seed))
    return s


def run(s):
    case, g = s["case"], s["graph"]
    kind = case["kind"]
    if kind == "walks":
        n, out = case["walks"], s["out"]
        if case["sink"] == "count":
            out.zero_()
            g.walk_device(s["params"], s["walks"], n, counts=out)
            return out
        if case["sink"] == "closure":
            out.zero_()
            g.walk_device(s["params"], s["walks"], n, closure=out)
            return out
        out.fill_(-1)
        g.walk_device(s["params"], s["walks"], n, paths=out, plen=s["lens"])
        return out, s["lens"]
    if kind == "pools":
        g.run_pools(s["params"], s["words"].data_ptr(), s["offsets"].data_ptr(), s["out"].data_ptr(), ids=s["ids"])
        return s["out"]
    if kind == "ppr":
        ids, counts, _ = g.ppr(s["params"], s["sources"], s["budgets"], 100, batched=case["batched"])
        return ids, counts
    if kind == "blocked":
        g.run(s["params"])
        return g.read_counts()
    if kind == "simrank":
        return g.simrank_batch(s["a"], s["b"], case["R"], case["L"], seed=s["seed"])
    if kind == "visits":
        return g.expected_visits(s["params"], s["source"])
    tickets = [s["server"].submit(int(v), int(b), stream=i)
               for i, (v, b) in enumerate(zip(s["sources"], s["budgets"]))]
    lists = [s["server"].wait(t)[:2] for t in tickets]
    return np.stack([x for x, _ in lists]), np.stack([x for _, x in lists])


def _visits_per_walk(case) -> float:
    """Visits of one walk: a draw continues with probability 0.85; about a third of R-MAT's moves meet a vertex
    without out-edges, where the stop rules end too."""
    L, rule = case["L"], case.get("rule", "restart")
    if rule in ("jump",):
        return L
    if rule == "restart":
        return max(1, L - 1)
    go = 0.85 if rule == "ppr" else 0.85 * 0.67
    return 1 / (1 - go) if rule == "prob" else (1 - go ** L) / (1 - go)


def work(case) -> dict:
    """Bytes: a 32-byte sector for every move (the next vertex), the walks in and the results out.
    Operations: the ten rounds of a draw's block, two products each, for every visit."""
    kind, nv = case["kind"], 1 << case["scale"]
    if kind == "visits":
        hops = max(1, case["L"] - 1) if case["rule"] == "restart" else case["L"]
        # the edges, the row pointer and the hop's input and output vectors, every hop
        return {"bytes": hops * (nv * (EF * 4 + 8 + 16)) + nv * 8, "flops": hops * nv * EF}
    if kind == "simrank":
        walks, visits = 2 * case["pairs"] * case["R"], max(1, case["L"] - 1)
        # every walk's visits once, and a comparison of each position's visits
        return {"bytes": walks * visits * 32 + case["pairs"] * (case["L"] * 8 + 16), "flops": walks * visits * 20}
    if kind == "ppr":
        b = case["budget"]
        mean = (b - 100) / math.log(b / 100) if case["spread"] and b > 101 else b
        walks, out = case["queries"] * mean, case["queries"] * 800
    elif kind == "serve":
        walks, out = case["queries"] * 298, case["queries"] * 800
    else:
        walks = case["walks"]
        out = {"path": walks * (case["L"] + 1) * 4, "closure": 8}.get(case.get("sink"), nv * 4)
    visits = _visits_per_walk(case)
    per_walk = {"walks": 16, "pools": 8, "blocked": 12}.get(kind, 0)
    return {"bytes": walks * ((visits - 1) * 32 + per_walk) + out, "flops": walks * visits * 20}


def _philox(c0, c1, seed: int):
    """Words 0 and 1 of Philox4x32-10 with counter (c0, c1, 0, 0), shifted right by one."""
    mask = 0xFFFFFFFF
    c2 = torch.zeros_like(c0)
    c3 = torch.zeros_like(c0)
    k0, k1 = seed & mask, (seed >> 32) & mask
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = (((p1 >> 32) & mask) ^ c1 ^ k0), p1 & mask, (((p0 >> 32) & mask) ^ c3 ^ k1), p0 & mask
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c0 >> 1, c1 >> 1


def _exact_visits(case, seed: int):
    rowptr, colidx = _csr(case["scale"], seed)
    deg = rowptr[1:] - rowptr[:-1]
    nv, src = len(deg), int(torch.argmax(deg))
    q, rule = ((1 << 31) - THRESHOLD) / (1 << 31), case["rule"]
    x = torch.zeros(nv, dtype=torch.float64, device="cuda")
    x[src] = 1.0
    visits = torch.zeros_like(x)
    edges = deg > 0
    for _ in range(max(1, case["L"] - 1) if rule == "restart" else case["L"]):
        visits += x
        share = torch.where(edges, x * q / deg.clamp(min=1), 0.0)
        y = torch.zeros_like(x).index_add_(0, colidx, torch.repeat_interleave(share, deg))
        fail = torch.where(edges, x * (1 - q), x)
        if rule == "restart":
            y[src] += fail.sum()
        elif rule == "ppr":
            y[src] += fail[~edges].sum()
        elif rule == "jump":
            y += fail.sum() / nv
        x = y
    return visits.cpu().numpy()


def _exact_simrank(case, seed: int):
    """Scores of every pair, walked and compared in torch (restart walks keyed on their vertex and hop)."""
    rowptr, colidx = _csr(case["scale"], seed)
    deg = rowptr[1:] - rowptr[:-1]
    a, b = _pairs(case, rowptr, seed)
    R, L = case["R"], case["L"]
    verts, inverse = np.unique(np.r_[a, b], return_inverse=True)
    src = torch.from_numpy(verts.astype(np.int64)).cuda().repeat_interleave(R)
    v, hop = src.clone(), (torch.arange(R, device="cuda") * L).repeat(len(verts))
    paths = torch.full((len(verts) * R, L), -1, dtype=torch.int64, device="cuda")
    for k in range(L - 1):  # a segment ends when it reaches hop % L == L - 1
        paths[:, k] = v
        d0, d1 = _philox(src, hop + k, seed)
        go = (deg[v] > 0) & (d0 >= THRESHOLD)
        at = rowptr[v] + torch.where(go, d1 % deg[v].clamp(min=1), 0)
        v = torch.where(go, colidx[at.clamp(max=len(colidx) - 1)], src)
    paths = paths.view(len(verts), R, L)
    scores = []
    for p, q in zip(inverse[: len(a)], inverse[len(a):]):
        open_pairs = torch.ones(R, R, dtype=torch.bool, device="cuda")
        meet = []
        for k in range(L):
            x, y = paths[p, :, k], paths[q, :, k]
            now = open_pairs & (x[:, None] == y[None, :]) & (x[:, None] >= 0)
            meet.append(now.sum())
            open_pairs &= ~now
        meet = torch.stack(meet).double()
        scores.append((meet * 0.8 ** torch.arange(L, device="cuda", dtype=torch.float64)).sum() / (R * R))
    return torch.stack(scores).cpu().numpy()


def exact(case, seed: int):
    if case["kind"] == "visits":
        return _exact_visits(case, seed)
    if case["kind"] == "simrank":
        return _exact_simrank(case, seed), None  # the counts are whole numbers
    return None
