"""The work that programs give this library, as cases to time and to compare.

Every case goes through the Python binding (mce_b200), whose calls are the C
ABI's.  Graphs come from the library's seeded generators with the parameters
of bench.py, smaller and larger: Erdos-Renyi with planted cliques, R-MAT,
Barabasi-Albert with planted cliques, and batches of Chung-Lu graphs.  The
answers are whole numbers (clique counts by size, peel rounds, core numbers),
so they are compared exactly.

Kinds of a case ("kind"):
  count       a resident graph: peel, orient, search (mce_count)
  file        a .bel file straight to the device, counted, freed: the command
              line's work
  order       the degeneracy order alone (mce_degeneracy)
  batch       a resident batch of graphs (mce_batch_count)
  batch_host  a batch in pinned host memory, copied and counted in one call
              (mce_batch_count_host)
  serve       a burst of 2-hop ego-graph requests to an open session
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "mce-gpu_b200"))
import mce_b200 as mce  # noqa: E402

MODEL = os.path.join(_ROOT, "mce-gpu_b200", "data", "cost_mlp_batch.f32")
SCHED = {"plain": mce.SCHED_PLAIN, "degree": mce.SCHED_DEGREE, "learned": mce.SCHED_LEARNED}


def listed():
    return [
        # one small graph per call, as a program that looks at many communities in
        # turn does: launches and synchronisations are most of the call
        {"name": "er-200", "kind": "count", "graph": "er", "n": 200, "degree": 10.0, "planted": 2,
         "px": False},
        # an ordinary small graph: bench.py's Erdos-Renyi workload
        {"name": "er-10k", "kind": "count", "graph": "er", "n": 10000, "degree": 20.0,
         "planted": 20, "px": False},
        # a large sparse graph with a power-law tail: bench.py's Barabasi-Albert
        # workload at a quarter of its size
        {"name": "ba-1m", "kind": "count", "graph": "ba", "n": 1000000, "m": 8, "planted": 50,
         "px": False},
        # a dense core whose search trees are most of the call (wide roots): bench.py's
        # R-MAT workload
        {"name": "rmat-13", "kind": "count", "graph": "rmat", "scale": 13, "edge_factor": 16,
         "px": False},
        # the same kind of graph with pivots from outside the subgraph (-i px)
        {"name": "rmat-12-px", "kind": "count", "graph": "rmat", "scale": 12, "edge_factor": 16,
         "px": True},
        # a graph file counted once, as the command line does
        {"name": "file-ba-100k", "kind": "file", "graph": "ba", "n": 100000, "m": 8, "planted": 20,
         "px": False},
        # the degeneracy order of a graph, for programs that only rank vertices
        {"name": "order-rmat-17", "kind": "order", "graph": "rmat", "scale": 17,
         "edge_factor": 16, "px": False},
        # a batch of a few small graphs in one call
        {"name": "batch-64", "kind": "batch", "graphs": 64, "n_max": 2048, "sched": "plain"},
        # bench.py's batch of mixed sizes, a quarter of its graphs, in its root order
        {"name": "batch-1024", "kind": "batch", "graphs": 1024, "n_max": 16384, "sched": "degree"},
        # the root order that the shipped cost model gives
        {"name": "batch-256-learned", "kind": "batch", "graphs": 256, "n_max": 16384,
         "sched": "learned"},
        # the batch arriving from pinned host memory, bench.py's end-to-end path
        {"name": "host-1024", "kind": "batch_host", "graphs": 1024, "n_max": 16384,
         "sched": "degree"},
        # serving at capacity: bench.py's requests, all at once
        {"name": "serve-ba-200k", "kind": "serve", "graph": "ba", "n": 200000, "m": 8,
         "planted": 20, "requests": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["count", "count", "count", "file", "order", "batch", "batch", "batch_host",
                       "serve"])
    if kind in ("batch", "batch_host"):
        return {"kind": kind, "graphs": _log_int(rng, 8, 900),
                "n_max": _log_int(rng, 512, 16384),
                "sched": rng.choice(["plain", "degree", "learned"] if kind == "batch"
                                    else ["plain", "degree"])}
    if kind == "serve":
        return {"kind": kind, "graph": "ba", "n": _log_int(rng, 20000, 200000),
                "m": rng.choice([4, 6, 8]), "planted": rng.randint(0, 20),
                "requests": _log_int(rng, 256, 4096)}
    graph = rng.choice(["er", "ba", "rmat"])
    if graph == "er":
        return {"kind": kind, "graph": "er", "n": _log_int(rng, 100, 200000),
                "degree": round(rng.uniform(6.0, 40.0), 2), "planted": rng.randint(1, 20),
                "px": kind == "count" and rng.random() < 0.2}
    if graph == "ba":
        top = 800000 if kind == "count" else 150000
        return {"kind": kind, "graph": "ba", "n": _log_int(rng, 1000, top),
                "m": rng.choice([3, 5, 8, 12]), "planted": rng.randint(1, 40),
                "px": kind == "count" and rng.random() < 0.2}
    return {"kind": kind, "graph": "rmat", "scale": rng.randint(8, 17 if kind == "order" else 12),
            "edge_factor": rng.randint(6, 16), "px": kind == "count" and rng.random() < 0.4}


def _host_graph(case, seed):
    if case["graph"] == "er":
        n = case["n"]
        return mce.gen_er(n, min(1.0, case["degree"] / n), seed, case["planted"], 6, 12)
    if case["graph"] == "ba":
        return mce.gen_ba(case["n"], case["m"], seed, case["planted"], 20, 60)
    return mce.gen_rmat(case["scale"], case["edge_factor"], 0.57, 0.19, 0.19, seed)


def _host_batch(case, seed):
    return mce.gen_chung_lu_batch(case["graphs"], 64, case["n_max"], 2.3, 8.0, 32.0, 5, 5, 40, seed)


class _File:
    """A .bel file that is removed with the state that holds it."""

    def __init__(self, hg):
        fd, self.path = tempfile.mkstemp(suffix=".bel")
        os.close(fd)
        mce.bel_write(self.path, hg)

    def __del__(self):
        try:
            os.unlink(self.path)
        except OSError:
            pass


def _opts(case):
    o = {"sched": SCHED[case.get("sched", "plain")]}
    if case.get("px"):
        o["induced"] = mce.INDUCED_PX
    return o


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("batch", "batch_host"):
        hb = _host_batch(case, seed)
        s["opts"] = _opts(case)
        if case["sched"] == "learned":
            s["opts"]["model"] = mce.Model()
            s["opts"]["model"].load(MODEL)
        s["batch"] = mce.Batch(hb)
        if kind == "batch_host":
            s["host"] = [torch.from_numpy(x).pin_memory()
                         for x in (hb.row_ptr, hb.col, hb.vtx_offsets, hb.arc_offsets)]
            s["graphs"] = hb.num_graphs
        return s
    hg = _host_graph(case, seed)
    if kind == "file":
        s["file"], s["opts"] = _File(hg), _opts(case)
        return s
    s["graph"] = mce.Graph.from_host(hg)
    if kind == "count":
        s["opts"] = _opts(case)
    elif kind == "serve":
        rng = np.random.default_rng(seed)
        s["seeds"] = rng.integers(0, hg.n, case["requests"])
        # a session that leaves the GPU as soon as the burst is answered
        s["serve"] = mce.Serve(s["graph"], ego_cap=16384, ring=4096, idle_ms=1)
    return s


def run(s):
    kind = s["kind"]
    if kind == "count":
        r = s["graph"].count(**s["opts"])
        return {"total": r.total, "hist": r.hist, "degeneracy": r.stats["degeneracy"]}
    if kind == "file":
        with mce.Graph.load_bel(s["file"].path) as g:
            r = g.count(**s["opts"])
        return {"total": r.total, "hist": r.hist, "degeneracy": r.stats["degeneracy"]}
    if kind == "order":
        prio, core, degeneracy = s["graph"].degeneracy()
        return {"prio": prio, "core": core, "degeneracy": degeneracy}
    if kind == "batch":
        r = s["batch"].count(**s["opts"])
    elif kind == "batch_host":
        r = s["batch"].count_host(*[t.data_ptr() for t in s["host"]], s["graphs"], **s["opts"])
    else:
        res, _ = s["serve"].run(s["seeds"])
        return {k: np.ascontiguousarray(res[k]) for k in ("count", "status", "ego_n", "ego_arcs")}
    return {"total": r.total, "per_graph": r.per_graph, "hist": r.hist}


def _size(case):
    """Expected vertices and arcs of a case's input."""
    if case["kind"] in ("batch", "batch_host"):
        lo, hi = 64.0, float(max(case["n_max"], 65))
        n = case["graphs"] * (hi - lo) / math.log(hi / lo)
        return n, 18.0 * n
    if case["graph"] == "er":
        return case["n"], case["n"] * case["degree"]
    if case["graph"] == "ba":
        return case["n"], 2.0 * case["n"] * case["m"]
    n = 2.0 ** case["scale"]
    return n, 1.6 * n * case["edge_factor"]


def work(case):
    """The graph's CSR read once and the answer written once.  (The search
    itself has no closed form: its tree depends on the graph.)"""
    n, m = _size(case)
    b = 4.0 * (n + 1) + 4.0 * m
    if case["kind"] == "order":
        b += 8.0 * n
    elif case["kind"] == "file":
        b = 24.0 * m + 8.0 * 4096
    elif case["kind"] == "serve":
        # each request's ego graph: its members' rows, about a thousand of them here
        b = case["requests"] * 1000.0 * 4.0 * (2.0 * case["m"] + 1.0)
    else:
        b += 8.0 * 4096
    return {"bytes": b, "flops": 0.0}


def tolerance(case):
    return "exact"


def exact(case, seed):
    """Plain Python for the graphs that are small enough: the degeneracy
    order's core numbers, and one pivoted Bron-Kerbosch search per vertex over
    its later neighbours, sets as integers' bits."""
    if case["kind"] != "count" or case["graph"] != "er" or case["n"] > 20000:
        return None
    hg = _host_graph(case, seed)
    adj = [set(hg.col[hg.row_ptr[v]:hg.row_ptr[v + 1]].tolist()) for v in range(hg.n)]
    deg = [len(a) for a in adj]
    buckets = [set() for _ in range(max(deg) + 1)]
    for v, d in enumerate(deg):
        buckets[d].add(v)
    rank, degeneracy, k = [-1] * hg.n, 0, 0
    for i in range(hg.n):
        k = max(k - 1, 0)
        while not buckets[k]:
            k += 1
        v = buckets[k].pop()
        degeneracy = max(degeneracy, k)
        rank[v] = i
        for u in adj[v]:
            if rank[u] < 0:
                buckets[deg[u]].remove(u)
                deg[u] -= 1
                buckets[deg[u]].add(u)
    hist = np.zeros(mce.HIST_MAX, np.uint64)
    for v in range(hg.n):
        stack = [({u for u in adj[v] if rank[u] > rank[v]}, {u for u in adj[v] if rank[u] < rank[v]},
                  1)]
        while stack:
            P, X, size = stack.pop()
            if not P:
                if not X and size > 1:
                    hist[size] += np.uint64(1)
                continue
            pivot = max(P | X, key=lambda u: len(P & adj[u]))
            for u in list(P - adj[pivot]):
                stack.append((P & adj[u], X & adj[u], size + 1))
                P.remove(u)
                X.add(u)
    return {"total": int(hist.sum()), "hist": hist, "degeneracy": degeneracy}
