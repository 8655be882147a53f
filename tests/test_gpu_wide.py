"""The wide launches together (65 to 128, 129 to 256 and more later
neighbours), on roots whose trees branch, share subtrees and go deeper than the
frames in shared memory: per-root counts and tree sizes against the oracle."""
import numpy as np
import pytest

import mce_b200 as mce
import oracle
from graphs import complete, core
from test_gpu_lanes import together
from test_gpu_rows import hub

pytestmark = pytest.mark.gpu

CORES = [core(50, 25, 6, 50, 3), core(110, 24, 6, 40, 5), core(160, 40, 5, 30, 7)]
GRAPHS = {
    "cores up to 240": lambda: CORES,
    "beside a clique of 460": lambda: CORES + [mce.gen_rmat(12, 16, 0.57, 0.19, 0.19, 3), complete(460)],
    "beside a clique of 1000": lambda: CORES + [mce.gen_rmat(11, 16, 0.57, 0.19, 0.19, 5), complete(1000)],
    "a core of 680": lambda: CORES + [core(580, 50, 4, 8, 9)],
}
SHARED = {"donate_after": 1, "donate_threshold": 4}


@pytest.mark.parametrize("name", GRAPHS)
@pytest.mark.parametrize("kw", [{}, SHARED, {"worker_list": mce.WL_OFF}, dict(SHARED, cuda_graph=1)], ids=str)
def test_roots_match_oracle(name, kw):
    g = together(GRAPHS[name]())
    tot, hist, rc_o, rn_o = oracle.roots(g)
    with mce.Graph.from_host(g) as dg:
        for _ in range(2):
            r = dg.count(log_roots=True, **kw)
            assert r.total == tot and np.array_equal(r.hist, hist)
            assert np.array_equal(dg.root_counts(), rc_o)
            assert np.array_equal(dg.root_log(), rn_o)
            assert (r.stats["donations"] > 0) == ("worker_list" not in kw)
        r = dg.count(x_pivot=1, log_roots=True, **kw)
        assert r.total == tot and np.array_equal(dg.root_counts(), rc_o)
        assert dg.count(level=mce.LEVEL_L2, **kw).total == tot


@pytest.mark.parametrize("kw", [{}, SHARED, {"worker_list": mce.WL_OFF}], ids=str)
def test_wide_class_of_narrow_roots_only(kw):
    """Hubs with more than 16,384 earlier and few later neighbours: the wide
    class, in a graph without a root of more than 64 later neighbours."""
    g = hub(17500, 20, 3)
    tot, hist, rc_o, rn_o = oracle.roots(g)
    with mce.Graph.from_host(g) as dg:
        for graph in (0, 1):
            r = dg.count(log_roots=True, cuda_graph=graph, **kw)
            assert r.stats["class_roots"][2] > 0 and 16 < r.stats["max_later_degree"] <= 64
            assert r.total == tot and np.array_equal(r.hist, hist)
            assert np.array_equal(dg.root_counts(), rc_o)
            assert np.array_equal(dg.root_log(), rn_o)
        assert dg.count(x_pivot=1, **kw).total == tot


@pytest.mark.parametrize("name,threshold", [("cores up to 240", 129), ("a core of 680", 257)])
def test_donations_of_every_wide_launch(name, threshold):
    """Subtrees of so many candidates come from the first launches only."""
    with mce.Graph.from_host(together(GRAPHS[name]())) as dg:
        for graph in (0, 1):
            r = dg.count(donate_after=1, donate_threshold=threshold, cuda_graph=graph)
            assert r.stats["donations"] > 0


@pytest.mark.parametrize("kw", [{}, SHARED, {"x_pivot": 1, "donate_after": 1}], ids=str)
def test_batches_match_oracle(kw):
    gs = GRAPHS["beside a clique of 1000"]() + CORES
    want = [oracle.count(g)[0] for g in gs]
    vo = np.concatenate([[0], np.cumsum([g.n + 1 for g in gs])]).astype(np.int64)
    ao = np.concatenate([[0], np.cumsum([g.m for g in gs])]).astype(np.int64)
    hb = mce.HostGraph(np.concatenate([g.row_ptr[:g.n + 1] for g in gs]).astype(np.int32),
                       np.concatenate([g.col for g in gs]).astype(np.int32), int(vo[-1]), int(ao[-1]),
                       len(gs), vo, ao)
    assert hb.m >= 1 << 20  # counted part by part from the host
    with mce.Batch(hb) as db:
        for _ in range(2):
            assert db.count(**kw).per_graph.tolist() == want
            r = db.count_host(hb.row_ptr.ctypes.data, hb.col.ctypes.data, vo.ctypes.data,
                              ao.ctypes.data, len(gs), **kw)
            assert r.per_graph.tolist() == want
