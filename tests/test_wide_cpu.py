"""The wide engine's kernels on the CPU: trees, frames and the tasks that its
warps share, for every size that the widest root of a graph gives a task."""
import numpy as np
import pytest

import emulate
import oracle
from graphs import core

# roots of 65 to 128 and of 129 to 256 later neighbours
GRAPHS = {2: dict(clique=50, chain=25, missing=6, around=50, seed=3),
          4: dict(clique=110, chain=24, missing=6, around=40, seed=5)}


def search(W, dcap, xp, donate_after=1):
    g = core(**GRAPHS[W])
    prio, _, _ = oracle.peel(g)
    split, cs = oracle.orient(g, prio)
    rp = g.row_ptr[:g.n + 1]
    later = rp[1:] - split
    wide = np.nonzero(later > 64)[0]
    mine = wide[(later[wide] > 32 * W) & (later[wide] <= 64 * W)]
    rc, out, err = emulate.run("wide", dcap, W, int(xp), donate_after,
                               arrays=(rp, split, cs, wide.astype(np.int32)), timeout=120)
    assert rc == 0, err
    x = np.frombuffer(out, np.uint64)
    _, _, rc_o, rn_o = oracle.roots(g)
    assert len(mine) > 20 and rn_o[mine].max() > 100
    return x[:g.n][mine], rc_o[mine], x[g.n:2 * g.n][mine], rn_o[mine], int(x[-2]), int(x[-1])


@pytest.mark.parametrize("W", [2, 4])
@pytest.mark.parametrize("dcap", [40, 256, 448, 449, 640, 2048])
def test_shared_subtrees_whatever_the_widest_root(W, dcap):
    count, count_o, nodes, nodes_o, err, pushed = search(W, dcap, False)
    assert err == 0 and pushed > 20
    assert np.array_equal(count, count_o) and np.array_equal(nodes, nodes_o)


@pytest.mark.parametrize("W", [2, 4])
def test_frames_past_the_shared_ones_without_sharing(W):
    count, count_o, nodes, nodes_o, err, pushed = search(W, 256, False, 1 << 30)
    assert err == 0 and pushed == 0
    assert np.array_equal(count, count_o) and np.array_equal(nodes, nodes_o)


@pytest.mark.parametrize("W", [2, 4])
def test_outside_pivots(W):
    count, count_o, _, _, err, pushed = search(W, 600, True)
    assert err == 0 and pushed > 0
    assert np.array_equal(count, count_o)
