"""Counts on a device with hardly more memory free than the search needs: the
wide roots' rows, which it can do without, leave it that memory."""
import numpy as np
import pytest
import torch

import mce_b200 as mce
import oracle
from graphs import complete, core
from test_gpu_lanes import together

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(scope="module")
def graph():
    """Rows of some 300 MiB: 30,000 vertices, most of them earlier neighbours of
    every vertex of a clique of 300, beside branching cores."""
    n, k = 30000, 300
    rng = np.random.default_rng(1)
    i, j = np.triu_indices(k, 1)
    src = [i] + [np.full(24000, v) for v in range(k)]
    dst = [j] + [rng.choice(np.arange(k, n), 24000, replace=False) for _ in range(k)]
    hub = mce.from_edges(np.concatenate(src), np.concatenate(dst), n)
    return together([hub, core(110, 24, 6, 40, 5), complete(400)])


def rows_bytes(g):
    prio, _, _ = oracle.peel(g)
    split, _ = oracle.orient(g, prio)
    rp = g.row_ptr[:g.n + 1].astype(np.int64)
    d = rp[1:] - split
    return int((np.diff(rp) * ((d + 63) // 64) * 8)[d > 32].sum())


def host_batch(gs):
    vo = np.concatenate([[0], np.cumsum([g.n + 1 for g in gs])]).astype(np.int64)
    ao = np.concatenate([[0], np.cumsum([g.m for g in gs])]).astype(np.int64)
    return mce.HostGraph(np.concatenate([g.row_ptr[:g.n + 1] for g in gs]).astype(np.int32),
                         np.concatenate([g.col for g in gs]).astype(np.int32), int(vo[-1]),
                         int(ao[-1]), len(gs), vo, ao)


@pytest.mark.parametrize("kind", ["graph", "batch", "host batch"])
def test_count_fits_without_the_rows(graph, kind):
    rows = rows_bytes(graph)
    assert rows > 200 * MIB
    hb = host_batch([graph, core(50, 25, 6, 50, 3), complete(400)])
    count = {"graph": lambda g: g.count(), "batch": lambda g: g.count(),
             "host batch": lambda g: g.count_host(hb.row_ptr.ctypes.data, hb.col.ctypes.data,
                                                  hb.vtx_offsets.ctypes.data,
                                                  hb.arc_offsets.ctypes.data, hb.num_graphs)}[kind]
    opened = {"graph": lambda: mce.Graph.from_host(graph)}.get(kind, lambda: mce.Batch(hb))
    with opened() as g:
        before = free()
        want = count(g)
        needed = before - free() - rows  # slab, queues, sort scratch
    with opened() as g:
        ballast = torch.empty(free() - needed - rows // 2, dtype=torch.uint8, device="cuda")
        try:
            for _ in range(2):
                r = count(g)
                assert r.total == want.total and np.array_equal(r.hist, want.hist)
        finally:
            del ballast
            torch.cuda.empty_cache()
        assert count(g).total == want.total  # with memory again, and the rows
    extra = 0 if kind == "graph" else sum(oracle.count(h)[0] for h in (core(50, 25, 6, 50, 3), complete(400)))
    assert want.total == oracle.count(graph)[0] + extra


def test_reload_takes_the_rows_memory(graph):
    """A larger graph into a handle whose rows leave it no memory."""
    larger = mce.gen_ba(1200000, 8, 5, 20, 20, 60)

    def reload(g, h):
        rp = np.ascontiguousarray(h.row_ptr[:h.n + 1], dtype=np.int32)
        col = np.ascontiguousarray(h.col, dtype=np.int32)
        g.reload_ptr(rp.ctypes.data, col.ctypes.data, h.n, h.m)
        torch.cuda.synchronize()

    with mce.Graph.from_host(graph) as g:
        total = g.count().total
        ballast = torch.empty(free() - 20 * MIB, dtype=torch.uint8, device="cuda")
        try:
            reload(g, larger)
        finally:
            del ballast
            torch.cuda.empty_cache()
        assert g.count().total == oracle.count(larger)[0]
        reload(g, graph)
        assert g.count().total == total
