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


@pytest.mark.parametrize("batch", [False, True])
def test_count_fits_without_the_rows(graph, batch):
    rows = rows_bytes(graph)
    assert rows > 200 * MIB
    opened = (lambda: mce.Batch(graph)) if batch else (lambda: mce.Graph.from_host(graph))
    with opened() as g:
        before = free()
        want = g.count()
        needed = before - free() - rows  # slab, queues, sort scratch
    with opened() as g:
        ballast = torch.empty(free() - needed - rows // 2, dtype=torch.uint8, device="cuda")
        try:
            for _ in range(2):
                r = g.count()
                assert r.total == want.total and np.array_equal(r.hist, want.hist)
        finally:
            del ballast
            torch.cuda.empty_cache()
        r = g.count()  # with memory again, and the rows
        assert r.total == want.total
        assert before - free() > 0
    assert want.total == oracle.count(graph)[0]
