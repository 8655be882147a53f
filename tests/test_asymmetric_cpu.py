"""CSRs that are not symmetric - a .bel file of one direction per edge passes
the reader's checks - have no defined counts, but no kernel may write outside
its arrays for them.  On the CPU, with symmetric graphs as the control."""
import numpy as np
import pytest

import emulate
import mce_b200 as mce
import oracle


def directed(n, rows):
    """A CSR from sorted rows of ids."""
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    return rp, np.concatenate([np.asarray(r, int) for r in rows])


def pointed_at(n, targets):
    """Every vertex points at `targets`, which point at one vertex each."""
    return directed(n, [[(v + 1) % n] if v in targets else [t for t in targets if t != v]
                        for v in range(n)])


def thinned(n, p, keep, seed):
    """A random graph of which each direction of an edge is kept with probability `keep`."""
    rng = np.random.default_rng(seed)
    a = np.triu(rng.random((n, n)) < p, 1)
    a = (a | a.T) & (rng.random((n, n)) < keep)
    return directed(n, [np.nonzero(r)[0] for r in a])


def forward(n, p, seed):
    a = np.triu(np.random.default_rng(seed).random((n, n)) < p, 1)
    a[:-1, -1] = True  # the last vertex's id sets n
    return directed(n, [np.nonzero(r)[0] for r in a[:-1]] + [[0]])


def repeated(targets=6, pointing=40, rest=30, arcs=32000):
    """Arcs repeated so often that the targets, whose rows are short, are pointed
    at by more arcs than a 16-bit degree holds beside its mark, before a rest of
    vertices of higher degree is peeled."""
    n = targets + pointing + rest
    return directed(n, [[targets]] * targets +
                    [np.repeat(np.arange(targets), arcs // pointing)] * pointing +
                    [np.repeat([v for v in range(n - rest, n) if v != n - rest + b], 200)
                     for b in range(rest)])


GRAPHS = {"pointed at": pointed_at(200, list(range(40, 80))), "thinned": thinned(300, 0.3, 0.6, 1),
          "thinned, dense": thinned(260, 0.9, 0.9, 2), "forward": forward(280, 0.5, 3)}


@pytest.mark.parametrize("name", list(GRAPHS) + ["repeated"])
def test_peel_stays_in_its_shared_memory(name):
    rp, col = repeated() if name == "repeated" else GRAPHS[name]
    rc, _, err = emulate.run("peel", arrays=(rp, col), timeout=60)
    assert rc == 0, err


def test_peel_of_a_symmetric_graph():
    g = mce.gen_er(301, 0.1, 4, 3, 10, 30)
    rc, out, err = emulate.run("peel", arrays=(g.row_ptr[:g.n + 1], g.col), timeout=60)
    assert rc == 0, err
    prio, core, _ = oracle.peel(g)
    x = np.frombuffer(out, np.uint32)
    assert np.array_equal(x[:g.n], prio) and np.array_equal(x[g.n:], core)


@pytest.mark.parametrize("name", GRAPHS)
@pytest.mark.parametrize("order", ["id", "reversed", "random"])
def test_row_pass_stays_in_its_regions(name, order):
    rp, col = GRAPHS[name]
    n = len(rp) - 1
    place = {"id": np.arange(n), "reversed": np.arange(n)[::-1],
             "random": np.random.default_rng(5).permutation(n)}[order]
    cs, split = [], []
    for v in range(n):
        r = col[rp[v]:rp[v + 1]]
        later = place[r] > place[v]
        split.append(rp[v] + int((~later).sum()))
        cs += [r[~later], r[later]]
    split = np.array(split)
    d = rp[1:] - split
    narrow, wide = np.nonzero((d > 0) & (d <= 32))[0], np.nonzero(d > 32)[0]
    rc, out, err = emulate.run("rows", arrays=(rp, split, np.concatenate(cs), narrow, wide), timeout=60)
    assert rc == 0, err
    assert int(out) == 0
