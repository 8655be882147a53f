"""Rows built before the search (enc.cu): per-root counts and tree sizes at the
edges of the rows' widths and of the list lengths, against the oracle."""
import numpy as np
import pytest

import mce_b200 as mce
import oracle

pytestmark = pytest.mark.gpu


def cliques(n, sizes, seed, degree=4.0, keep=0.97):
    """A sparse random graph with cliques of the given sizes planted on random
    vertices, so that roots of about those widths have trees of their own."""
    rng = np.random.default_rng(seed)
    g = mce.gen_er(n, degree / n, seed)
    src = [np.repeat(np.arange(n), np.diff(g.row_ptr[:n + 1]))]
    dst = [g.col]
    for s in sizes:
        v = rng.choice(n, s, replace=False)
        i, j = np.triu_indices(s, 1)
        kept = rng.random(len(i)) < (1.0 if s > 100 else keep)
        src.append(v[i][kept])
        dst.append(v[j][kept])
    return mce.from_edges(np.concatenate(src), np.concatenate(dst), n)


def hub(n, k, seed):
    """k vertices of a small clique adjacent to every other vertex: roots with
    few later and thousands of earlier neighbours."""
    g = mce.gen_er(n, 5.0 / n, seed)
    src = np.repeat(np.arange(n), np.diff(g.row_ptr[:n + 1]))
    h = np.repeat(np.arange(k), n)
    return mce.from_edges(np.concatenate([src, h]), np.concatenate([g.col, np.tile(np.arange(n), k)]), n)


@pytest.mark.parametrize("name,make", [
    ("rows of 31 to 34", lambda: cliques(700, [34, 35, 36, 37] * 2, 1)),
    ("rows of 62 to 66", lambda: cliques(1200, [64, 65, 66, 67, 68], 2, keep=0.993)),
    ("rows of 127 to 130", lambda: cliques(1500, [128, 129, 130, 131], 3)),
    ("rows of 255 to 258", lambda: cliques(2500, [256, 257, 258, 259], 4)),
    ("a row of 599", lambda: cliques(3000, [600, 24, 20], 5)),
    ("dense core", lambda: mce.gen_rmat(12, 16, 0.57, 0.19, 0.19, 3)),
    ("hubs", lambda: hub(6000, 9, 6)),
], ids=lambda x: x if isinstance(x, str) else "")
@pytest.mark.parametrize("kw", [{}, {"worker_list": mce.WL_OFF}, {"donate_after": 8}], ids=str)
def test_roots_match_oracle(name, make, kw):
    g = make()
    tot, hist, rc_o, rn_o = oracle.roots(g)
    with mce.Graph.from_host(g) as dg:
        for _ in range(3):  # rows and regions are rebuilt on every call
            r = dg.count(log_roots=True, **kw)
            assert r.total == tot and np.array_equal(r.hist, hist)
            assert np.array_equal(dg.root_counts(), rc_o)
            assert np.array_equal(dg.root_log(), rn_o)
        assert dg.count(x_pivot=1, **kw).total == tot
        assert dg.count(level=mce.LEVEL_L2, **kw).total == tot
