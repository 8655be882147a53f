"""The one-block peel at the edges of its range, against the oracle's peel."""
import numpy as np
import pytest

import mce_b200 as mce
import oracle
from graphs import build, complete, star

pytestmark = pytest.mark.gpu


def hubs(n, k, seed):
    """A sparse graph plus k vertices adjacent to all others: rows of n - 1
    arcs, more of them in one round than the block spreads over its warps."""
    base = mce.gen_er(n, 3.0 / n, seed)
    src = np.repeat(np.arange(n), np.diff(base.row_ptr[:n + 1]))
    h = np.repeat(np.arange(k), n)
    return mce.from_edges(np.concatenate([src, h]), np.concatenate([base.col, np.tile(np.arange(n), k)]), n)


@pytest.mark.parametrize("name,make", [
    ("one vertex", lambda: build(1, [])),
    ("one edge", lambda: build(2, [(0, 1)])),
    ("isolated and odd", lambda: build(7, [(1, 2), (2, 5), (5, 1), (5, 6)])),
    ("K300: every row long, one round", lambda: complete(300)),
    ("star: one long row", lambda: star(5000)),
    ("40 long rows in a round", lambda: hubs(2001, 40, 3)),
    ("rows of 256 and 257 arcs", lambda: build(520, [(0, i) for i in range(2, 258)] +
                                               [(1, i) for i in range(259, 516)])),
    ("16,383 vertices", lambda: mce.gen_er(16383, 9.0 / 16383, 5, 10, 6, 40)),
    ("16,384 vertices", lambda: mce.gen_ba(16384, 8, 5, 10, 20, 60)),
    ("16,385 vertices: grid", lambda: mce.gen_er(16385, 9.0 / 16385, 6)),
    ("R-MAT core", lambda: mce.gen_rmat(13, 16, 0.57, 0.19, 0.19, 3)),
    ("just above the arc limit: grid", lambda: mce.gen_er(3000, 0.06, 8)),
    ("grid, many rounds and long rows", lambda: mce.gen_rmat(15, 12, 0.57, 0.19, 0.19, 4)),
], ids=lambda x: x if isinstance(x, str) else "")
def test_peel_matches_oracle(name, make):
    g = make()
    prio_o, core_o, dg_o = oracle.peel(g)
    with mce.Graph.from_host(g) as dg:
        prio, core, d = dg.degeneracy()
        prio2, core2, _ = dg.degeneracy()
    assert d == dg_o
    assert np.array_equal(core, core_o) and np.array_equal(core2, core_o)
    assert np.array_equal(prio, prio_o) and np.array_equal(prio2, prio_o)
