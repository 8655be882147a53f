"""The lane engine at the edges of what a lane takes, and the roots and frames
it hands to the warp engine: per-root counts and tree sizes against the oracle."""
import numpy as np
import pytest

import mce_b200 as mce
import oracle
from graphs import complete, moon_moser

pytestmark = pytest.mark.gpu


def leaves(size, count):
    """A clique whose first vertex has `count` earlier neighbours, each adjacent
    to one more clique vertex: that many rows, of one bit."""
    i, j = np.triu_indices(size, 1)
    x = np.arange(size, size + count)
    return mce.from_edges(np.concatenate([i, x, x]),
                          np.concatenate([j, np.zeros(count, int), 1 + np.arange(count) % (size - 1)]))


def together(parts):
    """The disjoint union of graphs."""
    src, dst, n = [], [], 0
    for g in parts:
        src.append(np.repeat(np.arange(g.n), np.diff(g.row_ptr[:g.n + 1])) + n)
        dst.append(g.col.astype(np.int64) + n)
        n += g.n
    return mce.from_edges(np.concatenate(src), np.concatenate(dst), n)


@pytest.fixture(scope="module")
def mixed():
    """Enough small roots for the lane engine, cliques of 15 to 34 vertices,
    vertices with 31 to 66 earlier neighbours, and trees past a lane's share."""
    return together([mce.gen_er(1060000, 7.0 / 1060000, 7, 40, 6, 40)] +
                    [complete(k) for k in (15, 16, 17, 18, 31, 32, 33, 34)] +
                    [leaves(k, c) for k in (5, 16, 17, 30) for c in (31, 32, 33, 63, 64, 65, 300)] +
                    [moon_moser(k) for k in (5, 6, 8, 9, 10)] +
                    [mce.gen_er(60, 0.5, s) for s in range(40)] +
                    [mce.gen_rmat(10, 12, 0.57, 0.19, 0.19, 3)])


@pytest.mark.parametrize("kw", [{}, {"worker_list": mce.WL_OFF}, {"sched": mce.SCHED_DEGREE},
                                {"cuda_graph": 1}], ids=str)
def test_lanes_match_oracle(mixed, kw):
    tot, hist, rc_o, rn_o = oracle.roots(mixed)
    with mce.Graph.from_host(mixed) as dg:
        for _ in range(2):
            r = dg.count(log_roots=True, **kw)
            assert r.stats["class_roots"][0] >= 1000000
            assert r.total == tot and np.array_equal(r.hist, hist)
            assert np.array_equal(dg.root_counts(), rc_o)
            assert np.array_equal(dg.root_log(), rn_o)
            assert r.stats["tree_nodes"] == int(rn_o.sum())


def test_lanes_in_batches():
    hb = mce.gen_chung_lu_batch(960, 64, 16384, 2.3, 8.0, 32.0, 5, 5, 40, 21)
    _, _, rc, _ = oracle.roots(mce.union(hb))
    first = np.concatenate([[0], np.cumsum(np.diff(hb.vtx_offsets) - 1)])
    per = np.add.reduceat(rc, first[:-1])
    with mce.Batch(hb) as db:
        for sched in (mce.SCHED_PLAIN, mce.SCHED_DEGREE):
            assert np.array_equal(db.count(sched=sched).per_graph, per)
            arrays = [np.ascontiguousarray(x) for x in (hb.row_ptr, hb.col, hb.vtx_offsets, hb.arc_offsets)]
            r = db.count_host(*[x.ctypes.data for x in arrays], hb.num_graphs, sched=sched)
            assert np.array_equal(r.per_graph, per)
