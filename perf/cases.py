"""Timed cases: what programs that use ddp_gb300 ask of it.

listed() names the cases, draw() gives further ones of the same families and
ranges.  prepare() makes what a program holds before the call (a resident
graph, an engine, the query endpoints or update batches), run() is one pass
through the public entry points, exact() the same answer by a plain Dijkstra
where that is quick.

Families (the field "kind"):
  route      one query on a resident random digraph: the heuristic is built
             for its target, then the search runs (the reference's program:
             one source, one target)
  lib        the same through the LIB classes: GPU_A_Star with a heuristic
             array that the caller holds, get_path()
  maze       one corner-to-corner sized query on a grid maze, Manhattan bound
  mazepairs  a batch of maze queries, bidirectional A* on coordinates
  pairs      a batch of (source, target) pairs, bidirectional search on a
             random digraph (the headline workload at 4M nodes)
  hops       a batch with the engine's default heuristic (reverse BFS hops)
  landmark   a batch with the landmark (ALT) bound
  geo        a batch on a geometric graph (points joined to their nearest
             neighbours), bidirectional search
  dyn        one edge-update batch (half inserts, half deletes) of a resident
             dynamic search, and its new path
  serve      a live server: a batch of weight changes, then a burst of
             requests, drained

Graphs are fixed by the case (a program keeps its graph), queries and
updates come from the seed.  Weights up to 10^6 make shortest paths unique
for all practical purposes; where weights are small, equal-cost paths are
common and a case returns costs (and, on unit-weight mazes, path lengths),
not the path that a run happens to pick.
"""
import heapq
import math

import numpy as np

import ddp_gb300 as d


def listed():
    return [
        # a small road or dependency graph, one answer at a time: launches and round trips count
        {"name": "route_5k", "kind": "route", "n": 5000, "deg": 8, "wmax": 1000000, "K": 0},
        # the reference's own use: one query with K = 1024 queues on a 100,000-node graph
        {"name": "route_100k", "kind": "route", "n": 100000, "deg": 8, "wmax": 100, "K": 1024},
        # a C++ or Python program moved over from the LIB classes, heuristic array in hand
        {"name": "lib_250k", "kind": "lib", "n": 250001, "deg": 10, "wmax": 1000000, "K": 0},
        # a path planner on an occupancy grid
        {"name": "maze_511", "kind": "maze", "rows": 511, "cols": 511, "wall": 300},
        # several agents planned at once on a large grid
        {"name": "mazepairs_2048", "kind": "mazepairs", "rows": 2048, "cols": 2048, "wall": 300, "q": 16},
        # an interactive handful of queries
        {"name": "pairs_few_100k", "kind": "pairs", "n": 100000, "deg": 8, "wmax": 100, "q": 7},
        # the headline batch
        {"name": "pairs_4m", "kind": "pairs", "n": 4000000, "deg": 8, "wmax": 100, "q": 4096},
        # the batch engine as its defaults make it
        {"name": "hops_100k", "kind": "hops", "n": 100000, "deg": 8, "wmax": 100, "q": 300},
        # repeated queries on a fixed graph, with a landmark table built once
        {"name": "landmark_400k", "kind": "landmark", "n": 400000, "deg": 8, "wmax": 100, "q": 500},
        # a planar, road-like network
        {"name": "geo_1m", "kind": "geo", "n": 1000000, "q": 200},
        # a route kept current while the network changes
        {"name": "dyn_1m", "kind": "dyn", "n": 1000000, "deg": 10, "wmax": 1000000, "updates": 1000},
        # a routing service with live traffic
        {"name": "serve_400k", "kind": "serve", "n": 400000, "deg": 8, "wmax": 100, "q": 512, "updates": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["route", "lib", "maze", "mazepairs", "pairs", "pairs", "hops", "landmark", "geo", "dyn",
                       "serve"])
    c = {"kind": kind}
    if kind in ("maze", "mazepairs"):
        top = 700 if kind == "maze" else 2048
        c["rows"], c["cols"] = _log(rng, 64, top), _log(rng, 64, top)
        c["wall"] = rng.randint(100, 330)
        if kind == "mazepairs":
            c["q"] = _log(rng, 1, 64)
        return c
    if kind == "geo":
        c["n"], c["q"] = _log(rng, 20000, 1000000), _log(rng, 1, 200)
        return c
    top = {"route": 1000000, "lib": 500000, "pairs": 4000000, "hops": 200000, "landmark": 400000, "dyn": 1000000,
           "serve": 1000000}[kind]
    c["n"], c["deg"] = _log(rng, 50000 if kind == "dyn" else 2000, top), rng.randint(4, 12)
    c["wmax"] = 1000000 if kind in ("lib", "dyn") else rng.choice([20, 100, 1000, 1000000])
    if kind in ("pairs", "hops", "landmark", "serve"):
        c["q"] = _log(rng, 1, {"pairs": 4096, "hops": 300, "landmark": 500, "serve": 1024}[kind])
    if kind in ("route", "lib"):
        c["K"] = rng.choice([0, 0, 256, 1024, 8192])
    if kind in ("dyn", "serve"):
        c["updates"] = _log(rng, 10, 2000 if kind == "dyn" else 500)
    return c


# ---- inputs ---------------------------------------------------------------------
_host = {}   # graph of the current case (host CSR)
_dev = {}    # its device graph and engine, kept as a program keeps them


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


def _graph(case):
    k = _key(case)
    if k not in _host:
        _host.clear()
        if case["kind"] in ("maze", "mazepairs"):
            g = d.gen_maze(case["rows"], case["cols"], case["wall"] / 1000.0, 2002)
            g.extra["open"] = _reached(g, 0)
        elif case["kind"] == "geo":
            g = d.gen_geometric(case["n"], 6, 1 << 20, 100000, 5005)
        else:
            g = d.gen_random_chain(case["n"], case["deg"], 1, case["wmax"], 4004)
        _host[k] = g
    return _host[k]


def _reached(g, s):
    """Nodes that s reaches (level by level)."""
    seen = np.zeros(g.n, bool)
    seen[s] = True
    front = np.array([s])
    while len(front):
        lo, cnt = g.off[front], g.off[front + 1] - g.off[front]
        at = np.repeat(lo - np.cumsum(cnt) + cnt, cnt) + np.arange(int(cnt.sum()))
        nxt = np.unique(g.col[at])
        front = nxt[~seen[nxt]]
        seen[front] = True
    return np.flatnonzero(seen).astype(np.int32)


def _endpoints(case, seed):
    """(S, T) of the case's queries."""
    g, q = _graph(case), case.get("q", 1)
    rng = np.random.default_rng([seed, 11])
    if case["kind"] == "maze":
        # across the maze: a node of the first tenth to one of the last tenth
        o = g.extra["open"]
        k = max(1, len(o) // 10)
        return o[rng.integers(0, k, 1)], o[len(o) - 1 - rng.integers(0, k, 1)]
    if case["kind"] == "mazepairs":
        o = g.extra["open"]
        return o[rng.integers(0, len(o), q)], o[rng.integers(0, len(o), q)]
    if case["kind"] == "pairs":
        # uneven search depths: target hops log-uniform, clipped to what the graph has
        S, T, _ = d.gen_pairs(g, q, 4, 400, int(seed) % (1 << 31))
        return S, T
    return rng.integers(0, g.n, q).astype(np.int32), rng.integers(0, g.n, q).astype(np.int32)


def _updates(case, seed, batches):
    """Batches of half inserts of new random arcs, half deletes of arcs not yet deleted (the chain is kept), then
    the batches that take these back, last first: a program that runs on may start over."""
    g, m = _graph(case), case["updates"]
    rng = np.random.default_rng([seed, 12])
    ins = (m + 1) // 2
    dels = m - ins
    batches = max(1, min(batches, g.e // (4 * max(dels, 1))))
    src = np.repeat(np.arange(g.n, dtype=np.int32), np.diff(g.off))
    free = np.flatnonzero(g.protect_next()[src] != g.col)
    gone = rng.choice(free, batches * dels, replace=False, shuffle=False) if dels else free[:0]
    rng.shuffle(gone)
    out = []
    for b in range(batches):
        x = gone[b * dels:(b + 1) * dels]
        u = np.concatenate([rng.integers(0, g.n, ins, np.int32), src[x]])
        v = np.concatenate([rng.integers(0, g.n, ins, np.int32), g.col[x]])
        w = np.concatenate([rng.integers(1, case["wmax"] + 1, ins).astype(np.uint32), g.w[x]])
        f = np.concatenate([np.ones(ins, np.int32), np.zeros(dels, np.int32)])
        out.append((f, u, v, w))
    return out + [(1 - f, u, v, w) for f, u, v, w in reversed(out)]


# ---- what a program keeps -------------------------------------------------------
def _device(case):
    """(device graph, engine, server or GPU_Graph) of the case, made once."""
    k = _key(case)
    if k not in _dev:
        for dg, eng in _dev.values():
            if hasattr(eng, "close"):
                eng.close()
            dg.close()
        _dev.clear()
        g, kind, eng = _graph(case), case["kind"], None
        if kind == "lib":
            eng = d.GPU_Graph(d.Graph.from_csr(g))
        dg = eng.device if eng else d.DeviceGraph.from_csr(g)
        if kind == "landmark":
            dg.build_landmarks(64, seed=1, bits=8)
        if kind == "serve":
            eng = d.Server(dg, d.H_BIDIR, max_requests=1 << 22)
        elif kind in ("pairs", "geo"):
            eng = d.BatchEngine(dg, d.H_BIDIR)
        elif kind == "mazepairs":
            eng = d.BatchEngine(dg, d.H_BIDIR_MANHATTAN)
        elif kind == "hops":
            eng = d.BatchEngine(dg)
        elif kind == "landmark":
            eng = d.BatchEngine(dg, d.H_LANDMARK)
        _dev[k] = (dg, eng)
    return _dev[k]


class _Dynamic:
    """A resident dynamic search with its own graph (update batches change it)."""

    def __init__(self, case, seed):
        g = _graph(case)
        S, T = _endpoints(case, seed)
        self.kind = "dyn"
        self.graph = d.DeviceGraph.from_csr(g)
        self.search = d.DynamicSearch(self.graph, int(S[0]), int(T[0]), d.H_BFS_HOPS)
        self.batches, self.at = _updates(case, seed, 1500), 0

    def __del__(self):
        self.search.close()
        self.graph.close()


def prepare(case, seed):
    if case["kind"] == "dyn":
        return _Dynamic(case, seed)
    S, T = _endpoints(case, seed)
    dg, eng = _device(case)
    st = {"kind": case["kind"], "graph": dg, "engine": eng, "S": S, "T": T}
    if case["kind"] in ("route", "lib"):
        st["K"] = case["K"]
    if case["kind"] == "lib":
        h = dg.heuristic(int(T[0]), d.H_BFS_HOPS, want_values=True)
        st["search"] = d.GPU_A_Star(d.GPU_Dynamic_Graph(eng), int(S[0]), int(T[0]), case["K"])
        st["Hx"] = h.values
        h.close()
    if case["kind"] == "serve":
        # the same arcs in every state, with the state's own weights
        st["update"] = _traffic(case, seed)
    return st


def _traffic(case, seed):
    """Weight changes of one serving pass: the case's arcs, the seed's weights."""
    g, m = _graph(case), case["updates"]
    rows = np.flatnonzero(np.diff(g.off) > 0)
    u = np.random.default_rng(99).choice(rows, min(m, len(rows)), replace=False).astype(np.int32)
    v = g.col[g.off[u]]
    w = np.random.default_rng([seed, 13]).integers(1, case["wmax"] + 1, len(u)).astype(np.uint32)
    return np.full(len(u), 2, np.int32), u, v, w


def _padded(path):
    """The path as a row of fixed length (-1 after its end)."""
    row = np.full(max(256, len(path)), -1, np.int32)
    row[:len(path)] = path
    return row


def run(st):
    if not isinstance(st, dict):  # dyn
        b = st.batches[st.at % len(st.batches)]
        st.at += 1
        cost = st.search.update(*b)
        return [cost, _padded(st.search.path())]
    kind, dg, eng = st["kind"], st["graph"], st["engine"]
    if kind == "route":
        s, t = int(st["S"][0]), int(st["T"][0])
        h = dg.heuristic(t, d.H_BFS_HOPS, want_values=True)
        r = dg.solve(s, t, h, K=st["K"])
        h.close()
        return [r.cost, h.values]
    if kind == "lib":
        a = st["search"]
        a.set_huiristics(st["Hx"])
        return [_padded(a.get_path()), a.cost]
    if kind == "maze":
        s, t = int(st["S"][0]), int(st["T"][0])
        h = dg.heuristic(t, d.H_MANHATTAN)
        r = dg.solve(s, t, h)
        h.close()
        return [r.cost, len(r.path)]
    if kind == "mazepairs":
        cost, plen = eng.solve(st["S"], st["T"])
        return [cost, plen]
    if kind == "serve":
        eng.update(*st["update"])
        first = eng.submit(st["S"], st["T"])
        ids, costs, _, _ = eng.drain()
        out = np.empty(len(ids), np.int32)
        out[ids - first] = costs
        return out
    return eng.solve(st["S"], st["T"])[0]  # pairs, hops, landmark, geo: costs


# ---- the least work, and the answer by plain Dijkstra -----------------------------
def work(case):
    """Bytes of one pass: rows of the nodes that a search of the kind has to expand (8 bytes of row bounds, 8 per
    arc), plus inputs and outputs.  A bidirectional search of a random digraph meets after about 2 sqrt(n)
    expansions; a planar one covers about a tenth of the nodes between random ends; a reverse BFS reads every arc."""
    kind, q = case["kind"], case.get("q", 1)
    if kind in ("maze", "mazepairs"):
        cells = case["rows"] * case["cols"] * (1000 - case["wall"]) // 1000
        return {"bytes": q * (cells // 10 * (8 + 3 * 8) + 16), "flops": 0}
    if kind == "geo":
        return {"bytes": q * (case["n"] // 10 * (8 + 7 * 8) + 12), "flops": 0}
    n, row = case["n"], 8 + 8 * case["deg"]
    meet = 2 * int(math.sqrt(n)) * row
    whole = n * row
    if kind == "route":
        return {"bytes": whole + 4 * n + meet, "flops": 0}
    if kind == "lib":
        return {"bytes": 4 * n + meet, "flops": 0}
    if kind == "hops":
        return {"bytes": whole + q * (meet + 12), "flops": 0}
    if kind == "dyn":
        return {"bytes": case["updates"] * (16 + 2 * row) + meet, "flops": 0}
    return {"bytes": q * (meet + 12) + 16 * case.get("updates", 0), "flops": 0}  # pairs, landmark, serve


def _dijkstra(g, s, t):
    """(cost, path) of one query; INF and [] when t is unreachable."""
    off, col, w = g.off.tolist(), g.col.tolist(), g.w.tolist()
    dist, par, heap = {s: 0}, {s: -1}, [(0, s)]
    done = set()
    while heap:
        c, u = heapq.heappop(heap)
        if u in done:
            continue
        done.add(u)
        if u == t:
            path = [u]
            while par[path[-1]] >= 0:
                path.append(par[path[-1]])
            return c, path[::-1]
        for j in range(off[u], off[u + 1]):
            v, nc = col[j], c + w[j]
            if nc < dist.get(v, 1 << 62):
                dist[v] = nc
                par[v] = u
                heapq.heappush(heap, (nc, v))
    return d.INF, []


def _hops(g, t):
    """Reverse BFS hops x the smallest weight, -1 where t cannot be reached."""
    src = np.repeat(np.arange(g.n), np.diff(g.off))
    h = np.full(g.n, -1, np.int64)
    h[t], lvl = 0, 0
    while True:
        lvl += 1
        hit = src[(h[g.col] == lvl - 1) & (h[src] < 0)]
        if not len(hit):
            return h * np.where(h > 0, int(g.w.min()), 1)
        h[hit] = lvl


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dyn", "serve") or case.get("q", 1) > 8 or _graph(case).e > 3000000:
        return None
    g = _graph(case)
    S, T = _endpoints(case, seed)
    got = [_dijkstra(g, int(s), int(t)) for s, t in zip(S, T)]
    if kind == "route":
        return [got[0][0], _hops(g, int(T[0]))]
    if kind == "lib":
        return [_padded(got[0][1]), got[0][0]]
    if kind == "maze":
        return [got[0][0], len(got[0][1])]
    costs = np.array([c for c, _ in got], np.int32)
    return [costs, np.array([len(p) for _, p in got], np.int32)] if kind == "mazepairs" else costs
