"""CPU restatement of the bidirectional wave search: bucket lists behind a
window, a pile, lazy or eager labels, waves that open the next bucket while
they are narrow, the per-wave bounds that prune and stop.  Sequential, with
random order inside a wave; distances against Dijkstra."""
import heapq
import random

import pytest

INF = (1 << 31) - 1
NONE = 0xFFFFFFFF
LISTS = 32


def _graph(kind, n, wmax, rng):
    adj = [[] for _ in range(n)]
    if kind == "random":
        for u in range(n):
            for _ in range(rng.randint(0, 6)):
                adj[u].append((rng.randrange(n), rng.randint(0 if wmax < 5 else 1, wmax)))
    elif kind == "grid":
        side = int(n ** 0.5)
        for r in range(side):
            for c in range(side):
                for dr, dc in ((0, 1), (1, 0), (0, -1), (-1, 0)):
                    if 0 <= r + dr < side and 0 <= c + dc < side and rng.random() < 0.8:
                        adj[r * side + c].append(((r + dr) * side + c + dc, rng.randint(1, wmax)))
    else:  # two parts
        for u in range(n):
            for _ in range(4):
                v = rng.randrange(n // 2) + (n // 2 if u >= n // 2 else 0)
                adj[u].append((min(v, n - 1), rng.randint(1, wmax)))
    radj = [[] for _ in range(n)]
    for u in range(n):
        for v, w in adj[u]:
            radj[v].append((u, w))
    return adj, radj


def _dijkstra(adj, s, t):
    dist, heap = {s: 0}, [(0, s)]
    while heap:
        c, u = heapq.heappop(heap)
        if u == t:
            return c
        if c > dist[u]:
            continue
        for v, w in adj[u]:
            if c + w < dist.get(v, INF):
                dist[v] = c + w
                heapq.heappush(heap, (c + w, v))
    return None


def _search(adj, radj, s, t, width, room, fill, lazy, rng):
    if s == t:
        return 0
    rec = NONE if width <= 1 else (1 << 32) // width
    bucket = lambda k: (k * rec) >> 32  # noqa: E731
    edge = lambda b: min(NONE, ((b << 32) + rec - 1) // rec)  # noqa: E731
    label = ({}, {})
    lists = [[[] for _ in range(LISTS)] for _ in range(2)]
    pile, near, mu = [], [], NONE
    c = [bucket(0) - 1, bucket(0) - 1]
    lo = [c[0] + 1, c[1] + 1]
    lists[0][lo[0] % LISTS].append((s, 0))
    lists[1][lo[1] % LISTS].append((t, 0))
    if not lazy:
        label[0][s] = label[1][t] = 0
    lb = lim = None

    def to_lists(d, e, out):
        b = bucket(e[1])
        if 0 <= b - lo[d] < LISTS and len(lists[d][b % LISTS]) < room:
            lists[d][b % LISTS].append(e)
        else:
            out.append((d, e))

    for _ in range(200000):
        # plan
        lo = [c[0] + 1, c[1] + 1]
        nb = [next((lo[d] + i for i in range(LISTS) if lists[d][(lo[d] + i) % LISTS]), None) for d in (0, 1)]
        pm = [min([e[1] for dd, e in pile if dd == d], default=NONE) for d in (0, 1)]
        km = [min([e[1] for dd, e in near if dd == d], default=NONE) for d in (0, 1)]
        ed = [NONE if nb[d] is None else edge(nb[d]) for d in (0, 1)]
        lb = [min(km[d], pm[d], ed[d]) for d in (0, 1)]
        # the bound may never pass an open key
        for d in (0, 1):
            assert all(lb[d] <= e[1] for x in lists[d] for e in x)
        if NONE in lb or lb[0] + lb[1] >= mu:
            return None if mu == NONE else mu
        opened = []
        if len(near) < fill:
            if pm[0] < ed[0] or pm[1] < ed[1]:
                for d in (0, 1):
                    if nb[d] is None and pm[d] != NONE and pm[d] >= edge(lo[d]):
                        lo[d] = bucket(pm[d])
                    c[d] = lo[d] - 1
                lim = [edge(c[0] + 1), edge(c[1] + 1)]
                old, pile = pile, []
                for d, e in old:
                    if e[1] + lb[1 - d] >= mu:
                        continue
                    if e[1] >= lim[d]:
                        to_lists(d, e, pile)
                    else:
                        near.append((d, e))
                assert len(pile) < len(old)
                continue
            o = [sum(map(len, lists[d])) + sum(dd == d for dd, _ in pile) for d in (0, 1)]
            for d in (0, 1):
                if nb[d] is not None and (o[d] <= 2 * o[1 - d] + 64 or nb[1 - d] is None):
                    opened.append(d)
        wave = list(near)
        for d in opened:
            c[d] = lo[d] = nb[d]
            wave += [(d, e) for e in lists[d][c[d] % LISTS]]
            lists[d][c[d] % LISTS] = []
        assert wave
        lim = [edge(c[0] + 1), edge(c[1] + 1)]
        near = []
        rng.shuffle(wave)
        for d, (u, g) in wave:
            if g + lb[1 - d] >= mu:
                continue
            if lazy:
                if g >= label[d].get(u, INF):
                    continue
                label[d][u] = g
            elif label[d].get(u, INF) != g:
                continue
            for v, w in (adj, radj)[d][u]:
                ng = g + w
                if ng >= min(mu, INF):
                    continue
                mu = min(mu, ng + label[1 - d].get(v, INF) if v in label[1 - d] else mu)
                if label[d].get(v, INF) <= ng or ng + lb[1 - d] >= mu:
                    continue
                if not lazy:
                    label[d][v] = ng
                if ng < lim[d]:
                    near.append((d, (v, ng)))
                else:
                    to_lists(d, (v, ng), pile)
    raise AssertionError("the search did not end")


@pytest.mark.parametrize("lazy", [True, False])
@pytest.mark.parametrize("kind,n,wmax", [("random", 300, 100), ("random", 200, 3), ("grid", 225, 9),
                                         ("random", 150, 100000), ("parts", 200, 30)])
def test_wave_search_equals_dijkstra(kind, n, wmax, lazy):
    rng = random.Random(n + wmax + lazy)
    for rep in range(6):
        adj, radj = _graph(kind, n, wmax, rng)
        for _ in range(12):
            s, t = rng.randrange(n), rng.randrange(n)
            want = _dijkstra(adj, s, t)
            width = rng.choice([1, 2, max(1, wmax // 12), max(1, wmax // 4), 3 * wmax])
            got = _search(adj, radj, s, t, width, rng.choice([1, 3, 50]), rng.choice([1, 4, 32]), lazy, rng)
            assert got == want, (s, t, width)
