"""What the engine's users have it do, as measurable cases.

Every case is one call, or one short sequence of calls, through the Python
front end (``kcgpu_b200``) on synthetic graphs of the shapes the benchmark
configurations name: G(n, p), R-MAT, Chung-Lu with planted cliques and the
mixed batch of small graphs. ``kind`` says which part of the engine's surface
a case stands for:

  count     counting k-cliques of a graph that is resident and oriented (a
            user asks several questions about one graph);
  request   one graph of host arrays, built, oriented, counted and dropped
            (the one-request-per-call path);
  pipeline  the same from edges that are already in device memory;
  batch     many small graphs in one call, from host or device memory;
  local     per-vertex counts of a resident graph;
  multi     the counts for several k of a resident graph in one walk;
  analysis  core numbers and the truss support of every edge of a new graph;
  serve     a burst of requests to the request server, some of them about
            graphs it keeps resident.

All outputs are whole numbers, so every tolerance is "exact". Counts are
unsigned 128-bit integers and come back as four 32-bit limbs, lowest first.
"""
from __future__ import annotations

import math
import time

import numpy as np
import torch

import kcgpu_b200 as kc

_CTX = None


def _context() -> kc.Context:
    """The process's one context, as a program that uses the engine keeps it."""
    global _CTX
    if _CTX is None:
        torch.cuda.set_device(0)
        _CTX = kc.Context(0)
    return _CTX


# ---- the cases ----------------------------------------------------------------

def listed() -> list[dict]:
    return [
        # The smallest call: one count of the small G(2000, 0.01) configuration
        # (about 20k edges); launches and host latency are what it costs.
        dict(name="count_small", kind="count", graph="er", n=2000, p=0.01, orientation="degree", mode="orient",
             unit="node", part=8, encoding="bitmap", k=4),
        # A skewed graph, pivoting with edge units: the R-MAT configuration
        # (degeneracy orientation, partition 8, k = 5) at scale 17.
        dict(name="count_rmat", kind="count", graph="rmat", scale=17, ef=16.0, orientation="degen", mode="pivot",
             unit="edge", part=8, encoding="bitmap", k=5),
        # A power-law graph with planted cliques, pivoting with node units:
        # the Chung-Lu configuration with a quarter of its vertices.
        dict(name="count_chunglu", kind="count", graph="chunglu", n=1_000_000, mean=20.0, cap=12_500.0, cliques=50,
             orientation="degen", mode="pivot", unit="node", part=0, encoding="bitmap", k=6),
        # The list encoding with orientation listing, for graphs whose
        # neighbourhoods are kept as sorted lists instead of bitmaps.
        dict(name="count_list", kind="count", graph="rmat", scale=14, ef=16.0, orientation="degen", mode="orient",
             unit="node", part=8, encoding="list", k=4),
        # One request of the serving mix on its own: a host edge list is
        # built, oriented, counted once and dropped (mostly fixed costs).
        dict(name="request", kind="request", graph="rmat", scale=11, ef=10.3, orientation="degen", mode="pivot",
             unit="node", part=0, encoding="bitmap", k=8),
        # A large graph from device memory, end to end: CSR build, degeneracy
        # orientation and one count with a small k.
        dict(name="pipeline", kind="pipeline", graph="rmat", scale=18, ef=16.0, orientation="degen", mode="pivot",
             unit="edge", part=8, encoding="bitmap", k=4),
        # A batch of a few hundred mixed graphs from host arrays.
        dict(name="batch_host", kind="batch", graphs=400, n_min=50, n_max=5000, k_min=4, k_max=12,
             orientation="degree", device=False),
        # The headline: mixed graphs with the edge lists in device memory, a
        # quarter of the full batch of 10,000.
        dict(name="batch_device", kind="batch", graphs=2500, n_min=50, n_max=5000, k_min=4, k_max=12,
             orientation="degree", device=True),
        # Per-vertex counts (how many k-cliques contain each vertex).
        dict(name="local", kind="local", graph="rmat", scale=14, ef=12.0, orientation="degen", mode="pivot",
             unit="node", part=8, encoding="bitmap", k=4),
        # The clique profile of a resident graph: every k from 3 to 15.
        dict(name="multi", kind="multi", graph="rmat", scale=12, ef=13.5, orientation="degen", unit="node", k_min=3,
             k_max=15),
        # Core numbers and edge supports of a new graph.
        dict(name="analysis", kind="analysis", graph="rmat", scale=17, ef=16.0),
        # A burst of server requests, 30% of them about eight resident graphs.
        dict(name="serve", kind="serve", requests=256, max_edges=100_000, streams=2),
    ]


def draw(rng) -> dict:
    """One more case of the ranges above: sizes spread over their logarithm,
    odd vertex counts and edge counts among them."""
    kind = rng.choice(["count", "count", "count", "request", "pipeline", "batch", "batch", "local", "multi",
                       "analysis", "serve"])

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "count":
        which = rng.choice(["er", "rmat", "chunglu", "listing"])
        c = dict(kind=kind, orientation=rng.choice(["degree", "degen"]), unit=rng.choice(["node", "edge"]),
                 part=rng.choice([0, 4, 8, 16, 32]), encoding="bitmap")
        if which == "er":
            n = log_int(200, 20_000)
            c.update(graph="er", n=n, p=min(0.2, rng.uniform(10.0, 60.0) / n), mode=rng.choice(["orient", "pivot", "auto"]),
                     k=rng.randint(3, 6))
        elif which == "rmat":
            c.update(graph="rmat", scale=rng.randint(10, 16), ef=rng.uniform(6.0, 16.0), orientation="degen",
                     mode=rng.choice(["pivot", "auto"]), k=rng.randint(3, 5))
        elif which == "chunglu":
            n = log_int(30_000, 1_000_000)
            c.update(graph="chunglu", n=n, mean=rng.uniform(8.0, 20.0), cap=n / 80.0, cliques=rng.randint(5, 50),
                     orientation="degen", mode=rng.choice(["pivot", "auto"]), k=rng.randint(3, 6))
        else:
            c.update(graph="rmat", scale=rng.randint(9, 13), ef=rng.uniform(4.0, 16.0), orientation="degen",
                     mode=rng.choice(["orient", "pivot"]), encoding="list", k=rng.randint(3, 4))
        return c
    if kind in ("request", "multi"):
        edges = log_int(1_000, 60_000)  # the serving mix's sizes
        scale = max(1, math.ceil(math.log2(edges / 16)))
        c = dict(kind=kind, graph="rmat", scale=scale, ef=edges / (1 << scale), orientation="degen",
                 unit=rng.choice(["node", "edge"]))
        if kind == "request":
            c.update(mode=rng.choice(["pivot", "auto"]), part=rng.choice([0, 8]), encoding="bitmap",
                     k=rng.randint(3, 9))
        else:
            c.update(k_min=3, k_max=rng.randint(6, 15))
        return c
    if kind == "pipeline":
        return dict(kind=kind, graph="rmat", scale=rng.randint(12, 18), ef=rng.uniform(4.0, 16.0),
                    orientation=rng.choice(["degree", "degen"]), mode="pivot", unit=rng.choice(["node", "edge"]),
                    part=8, encoding="bitmap", k=rng.randint(3, 4))
    if kind == "batch":
        return dict(kind=kind, graphs=log_int(40, 2000), n_min=50, n_max=log_int(1500, 5000), k_min=4, k_max=12,
                    orientation=rng.choice(["degree", "degree", "degen"]), device=rng.random() < 0.5)
    if kind == "local":
        return dict(kind=kind, graph="rmat", scale=rng.randint(10, 14), ef=rng.uniform(5.0, 12.0),
                    orientation="degen", mode=rng.choice(["orient", "pivot"]), unit=rng.choice(["node", "edge"]),
                    part=8, encoding="bitmap", k=rng.randint(3, 4))
    if kind == "analysis":
        return dict(kind=kind, graph="rmat", scale=rng.randint(12, 17), ef=rng.uniform(4.0, 16.0))
    return dict(kind="serve", requests=log_int(32, 256), max_edges=log_int(10_000, 100_000), streams=rng.randint(1, 3))


# ---- inputs ---------------------------------------------------------------------

def _edges(case: dict, seed: int):
    """(src, dst, n) as host arrays; duplicates, loops and both directions as
    the generators give them."""
    if case["graph"] == "er":
        return kc.gen_er(case["n"], case["p"], seed).arrays()
    if case["graph"] == "rmat":
        return kc.gen_rmat(case["scale"], case["ef"], seed=seed).arrays()
    el = kc.gen_chung_lu(case["n"], 2.1, case["mean"], case["cap"], seed)
    el.plant_cliques(case["cliques"], 30, 60, seed + 1)
    return el.arrays()


def _distinct(case: dict) -> int:
    """Distinct edges of an analysis case's graph: R-MAT of these sizes has
    more (0.7 to 0.95 of the edges drawn)."""
    return int(0.6 * case["ef"] * (1 << case["scale"]))


def _up_to_distinct(s, d, n: int, m: int):
    """The edge list up to the edge that makes m distinct ones (so that the
    size of a per-edge result depends on the case alone); loops, duplicates
    and order stay as they were."""
    key = np.minimum(s, d).astype(np.int64) * n + np.maximum(s, d)
    key[s == d] = -1
    vals, first = np.unique(key, return_index=True)
    end = int(np.sort(first[vals >= 0])[m - 1]) + 1
    return s[:end], d[:end]


def _on_device(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def _requests(case: dict, seed: int):
    """The serving mix: R-MAT graphs with edges log-uniform in [1e3,
    max_edges], k in 3..12, 30% about one of eight resident graphs."""
    rng = np.random.default_rng(seed)

    def graph(i):
        e = int(np.exp(rng.uniform(np.log(1e3), np.log(case["max_edges"]))))
        scale = max(1, int(np.ceil(np.log2(e / 16))))
        return kc.gen_rmat(scale, e / (1 << scale), seed=seed * 1000 + i).arrays()

    resident = [graph(i) for i in range(8)]
    reqs = []
    for r in range(case["requests"]):
        k = int(rng.integers(3, 13))
        if rng.random() < 0.3:
            reqs.append((int(rng.integers(8)), None, k))
        else:
            reqs.append((-1, graph(100 + r), k))
    return resident, reqs


def prepare(case: dict, seed: int):
    ctx = _context()
    kind = case["kind"]
    st = {"case": case, "ctx": ctx}
    if kind == "batch":
        el = kc.gen_batch(case["graphs"], seed * 100_003 + 17, case["n_min"], case["n_max"], case["k_min"],
                          case["k_max"], pinned=not case["device"])
        off, nn, kk, _ = el.batch_meta()
        s, d, _ = el.arrays(copy=False)
        st.update(off=off, nn=nn, kk=kk)
        if case["device"]:
            st.update(src=_on_device(s), dst=_on_device(d))
        else:  # page-locked host arrays, owned by the list
            st.update(src=s, dst=d, owner=el)
    elif kind == "serve":
        resident, reqs = _requests(case, seed)
        srv = kc.Server(ctx, streams=case["streams"], orientation="degen")
        st.update(srv=srv, ids=[srv.put_graph(s, d, n) for s, d, n in resident], reqs=reqs)
    else:
        s, d, n = _edges(case, seed)
        if kind == "analysis":
            s, d = _up_to_distinct(s, d, n, _distinct(case))
        if kind == "request":
            st.update(src=s, dst=d, n=n)
        elif kind in ("pipeline", "analysis"):
            st.update(src=_on_device(s), dst=_on_device(d), edges=int(s.size), n=n)
        else:
            st["g"] = kc.Graph.from_edges(ctx, s, d, n).orient(case["orientation"])
    torch.cuda.synchronize()
    return st


# ---- one pass -------------------------------------------------------------------

def _limbs(counts) -> np.ndarray:
    return np.array([[(c >> s) & 0xFFFFFFFF for s in (0, 32, 64, 96)] for c in counts], dtype=np.int64)


def _count(g: kc.Graph, c: dict) -> int:
    return g.count(c["k"], mode=c["mode"], unit=c["unit"], part=c["part"], encoding=c["encoding"])


def run(st):
    c, ctx = st["case"], st["ctx"]
    kind = c["kind"]
    if kind == "count":
        return _limbs([_count(st["g"], c)])
    if kind == "request":
        with kc.Graph.from_edges(ctx, st["src"], st["dst"], st["n"]) as g:
            return _limbs([_count(g.orient(c["orientation"]), c)])
    if kind == "pipeline":
        with kc.Graph.from_edges_device(ctx, st["src"].data_ptr(), st["dst"].data_ptr(), st["edges"], st["n"]) as g:
            count = _count(g.orient(c["orientation"]), c)
            info = g.info()
        return {"count": _limbs([count]), "edges": info["m"], "max_out_degree": info["max_out_degree"]}
    if kind == "batch":
        ptrs = (st["src"].data_ptr(), st["dst"].data_ptr()) if c["device"] else None
        got = kc.batch_count(ctx, st["src"], st["dst"], st["off"], st["nn"], st["kk"], orientation=c["orientation"],
                             device_ptrs=ptrs)
        return np.array(got, dtype=np.int64)
    if kind == "local":
        return np.array(st["g"].count_local(c["k"], unit=c["unit"], part=c["part"], mode=c["mode"]), dtype=np.int64)
    if kind == "multi":
        return _limbs(st["g"].count_multi(range(c["k_min"], c["k_max"] + 1), unit=c["unit"]))
    if kind == "analysis":
        with kc.Graph.from_edges_device(ctx, st["src"].data_ptr(), st["dst"].data_ptr(), st["edges"], st["n"]) as g:
            core, top = g.kcore()
            return {"core": core.view(np.int32), "max_core": top, "support": g.truss_support().view(np.int32)}
    srv, ids = st["srv"], st["ids"]
    tickets = [srv.submit(ids[i], k) if i >= 0 else srv.submit_edges(g[0], g[1], g[2], k) for i, g, k in st["reqs"]]
    return _limbs([srv.wait(t)["count"] for t in tickets])


# ---- what a pass cannot do without -------------------------------------------------

def _size(case: dict) -> tuple[float, float]:
    """Expected (vertices, input edges) of a case's graph."""
    if case["graph"] == "er":
        return case["n"], 0.5 * case["p"] * case["n"] ** 2
    if case["graph"] == "rmat":
        return 1 << case["scale"], case["ef"] * (1 << case["scale"])
    return case["n"], 0.5 * case["mean"] * case["n"]


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "batch":
        # vertices log-uniform in [n_min, n_max], mean edge probability 0.027
        lo, hi = case["n_min"], case["n_max"]
        edges = case["graphs"] * 0.0135 * (hi * hi - lo * lo) / (2.0 * math.log(hi / lo))
        return {"bytes": 8.0 * edges + 32.0 * case["graphs"], "flops": 0.0}
    if kind == "serve":
        mean = (case["max_edges"] - 1e3) / math.log(case["max_edges"] / 1e3)
        return {"bytes": case["requests"] * (8.0 * mean + 16.0), "flops": 0.0}
    n, edges = _size(case)
    if kind in ("request", "pipeline"):  # the edge list in, a count out
        return {"bytes": 8.0 * edges + 16.0, "flops": 0.0}
    if kind == "analysis":  # the edge list in, a word per vertex and per edge out
        return {"bytes": 12.0 * _distinct(case) + 4.0 * n, "flops": 0.0}
    out = {"count": 16.0, "multi": 16.0 * 13, "local": 16.0 * n}[kind]
    return {"bytes": 4.0 * (edges + n + 1) + out, "flops": 0.0}  # the oriented CSR in


def tolerance(case: dict):
    return "exact"


# ---- the same numbers from plain torch ------------------------------------------------

class _TooLong(Exception):
    pass


class _Plain:
    """A simple graph as sorted edge keys on the GPU, oriented by degree, and
    its cliques listed level by level in bounded chunks."""

    def __init__(self, src, dst, n, limit_s=15.0):
        self.n, self.until = int(n), time.monotonic() + limit_s
        s = torch.from_numpy(src.astype(np.int64)).cuda()
        d = torch.from_numpy(dst.astype(np.int64)).cuda()
        keep = s != d
        s, d = s[keep], d[keep]
        key = torch.unique(torch.minimum(s, d) * self.n + torch.maximum(s, d))
        self.u, self.v = key // self.n, key % self.n
        deg = torch.bincount(torch.cat([self.u, self.v]), minlength=self.n)
        order = torch.argsort(deg, stable=True)
        rank = torch.empty_like(order)
        rank[order] = torch.arange(self.n, device=order.device)
        self.order = order  # rank -> vertex
        a, b = rank[self.u], rank[self.v]
        self.key, self.edge = torch.sort(torch.minimum(a, b) * self.n + torch.maximum(a, b))
        self.col = self.key % self.n
        self.rp = torch.searchsorted(self.key, torch.arange(self.n + 1, device=key.device) * self.n)
        self.deg = deg

    def has(self, a, b):
        q = a * self.n + b
        i = torch.searchsorted(self.key, q).clamp(max=self.key.numel() - 1)
        return self.key[i] == q, i

    def cliques(self, k, rows=None, chunk=1 << 24):
        """Yields blocks of k-cliques, rank labels ascending, one per row."""
        if rows is None:
            rows = torch.stack([self.key // self.n, self.col], 1)
        if time.monotonic() > self.until:
            raise _TooLong
        if rows.shape[0] == 0:
            return
        if rows.shape[1] == k:
            yield rows
            return
        last = rows[:, -1]
        more = self.rp[last + 1] - self.rp[last]
        ends = torch.cumsum(more, 0)
        at = 0
        while at < rows.shape[0]:
            base = int(ends[at - 1]) if at else 0
            to = max(at + 1, int(torch.searchsorted(ends, base + chunk, right=True)))
            cnt = more[at:to]
            i = torch.repeat_interleave(torch.arange(at, to, device=cnt.device), cnt)
            step = torch.arange(i.numel(), device=cnt.device) - (ends[i] - more[i] - base)
            w = self.col[self.rp[last[i]] + step]
            for j in range(rows.shape[1] - 1):
                ok, _ = self.has(rows[i, j], w)
                i, w = i[ok], w[ok]
            yield from self.cliques(k, torch.cat([rows[i], w[:, None]], 1), chunk)
            at = to

    def count(self, k):
        return self.n if k == 1 else self.key.numel() if k == 2 else sum(b.shape[0] for b in self.cliques(k))

    def local(self, k):
        got = torch.zeros(self.n, dtype=torch.int64, device=self.key.device)
        for b in self.cliques(k):
            got += torch.bincount(self.order[b.reshape(-1)], minlength=self.n)
        return got

    def support(self):
        got = torch.zeros(self.key.numel(), dtype=torch.int64, device=self.key.device)
        for b in self.cliques(3):
            for x, y in ((0, 1), (0, 2), (1, 2)):
                got += torch.bincount(self.edge[self.has(b[:, x], b[:, y])[1]], minlength=got.numel())
        return got

    def core(self):
        u, v = torch.cat([self.u, self.v]), torch.cat([self.v, self.u])
        order = torch.argsort(u, stable=True)
        v = v[order]
        rp = torch.zeros(self.n + 1, dtype=torch.int64, device=v.device)
        rp[1:] = torch.cumsum(self.deg, 0)
        deg, core = self.deg.clone(), torch.zeros_like(self.deg)
        alive = torch.ones(self.n, dtype=torch.bool, device=v.device)
        level = 0
        while bool(alive.any()):
            if time.monotonic() > self.until:
                raise _TooLong
            level = max(level, int(deg[alive].min()))
            front = torch.nonzero(alive & (deg <= level)).reshape(-1)
            core[front] = level
            alive[front] = False
            cnt = rp[front + 1] - rp[front]
            i = torch.repeat_interleave(torch.arange(front.numel(), device=v.device), cnt)
            step = torch.arange(i.numel(), device=v.device) - (torch.cumsum(cnt, 0) - cnt)[i]
            deg -= torch.bincount(v[rp[front[i]] + step], minlength=self.n)
        return core


def exact(case: dict, seed: int):
    """run()'s outputs from plain torch, or None where listing takes too long
    (the batches, the server's burst and graphs with very many cliques)."""
    if case["kind"] in ("batch", "serve"):
        return None
    s, d, n = _edges(case, seed)
    if case["kind"] == "analysis":
        s, d = _up_to_distinct(s, d, n, _distinct(case))
    try:
        g = _Plain(s, d, n)
        if case["kind"] == "analysis":
            core = g.core()
            return {"core": core, "max_core": int(core.max()), "support": g.support()}
        if case["kind"] == "local":
            return g.local(case["k"])
        if case["kind"] == "multi":
            return _limbs([g.count(k) for k in range(case["k_min"], case["k_max"] + 1)])
        count = _limbs([g.count(case["k"])])
        if case["kind"] == "pipeline":
            return {"count": count, "edges": g.key.numel(), "max_out_degree": None}
        return count
    except _TooLong:
        return None
