"""Whole weights whose sums do not fit 32 bits, in every form: such a graph, in
a union or alone, gets FP64 tables, whatever the other graphs of its union
hold.  Weights are small whole numbers or quarters times a power of two, one of
them 2^33 in one graph: every sum is exact (a vertex's in FP32 too), so
partitions equal the oracle's; Q to 1e-9, as in the other comparisons with it."""
import numpy as np
import pytest

import lvb200
import pyoracle

pytestmark = pytest.mark.gpu

BIG = 1 << 28  # a vertex's entries in its community add up past 2^32


def graph(scale, seed, large=0.0):
    # communities of 100, degrees of about 15, 45 and 90, five vertices of 400
    # to 1,800: rows of every table but the hubs', merges of a block each
    rng = np.random.default_rng(seed)
    n, size = 3000, 100
    v = np.repeat(np.arange(n), np.array([8, 22, 45])[np.arange(n) % 3])
    inside = rng.random(len(v)) < 0.85
    u = np.where(inside, v // size * size + rng.integers(0, size, len(v)),
                 rng.integers(0, n, len(v)))
    hubs = [(h * 500, 400 + 350 * h) for h in range(5)]
    v = np.concatenate([v] + [np.full(d, h) for h, d in hubs])
    u = np.concatenate([u] + [rng.choice(n, d, replace=False) for _, d in hubs])
    keep = u != v
    e = np.unique(np.minimum(u, v)[keep] * n + np.maximum(u, v)[keep])
    a, b = e // n, e % n
    w = (rng.integers(1, 4, len(e)) * scale).astype(np.float32)
    if large:
        w[np.flatnonzero((a // size == 7) & (b // size == 7))[0]] = large
    s, d, w = np.r_[a, b], np.r_[b, a], np.r_[w, w]
    o = np.lexsort((d, s))
    off = np.searchsorted(s[o], np.arange(n + 1)).astype(np.uint64)
    return n, off, d[o].astype(np.uint32), w[o]


GRAPHS = {
    "big": lambda: graph(BIG, 7),
    "one_large_weight": lambda: graph(4096, 7, large=2.0 ** 33),
}
UNIONS = {
    "alone": [GRAPHS["big"]],
    "with_small": [lambda: graph(1, 3), GRAPHS["big"], lambda: graph(3, 4)],
    "with_fractions": [lambda: graph(0.25, 3), GRAPHS["big"], lambda: graph(1, 4)],
    "one_large_weight": [lambda: graph(1, 3), GRAPHS["one_large_weight"]],
    # every graph's total fits, the union's does not
    "many_that_fit": [lambda s=s: graph(2048, s) for s in range(8)],
}


def _oracle(csr, rule, gain):
    n, off, col, w = csr
    return pyoracle.louvain(pyoracle.CSR(n, off, col, w.astype(np.float64)), 1e-6, rule=rule,
                            prec=gain, rows="sorted")


@pytest.mark.parametrize("rule,gain", [("py", "fp32"), ("cuda", "fp32"), ("py", "fp64")])
@pytest.mark.parametrize("form", ["batch", "serve"])
@pytest.mark.parametrize("union", sorted(UNIONS))
def test_union_equals_oracle(union, form, rule, gain):
    csrs = [make() for make in UNIONS[union]]
    graphs = [lvb200.Graph.from_csr(*c) for c in csrs]
    if form == "batch":
        with lvb200.Engine(rule=rule, gain=gain) as e:
            parts, q, levels, _ = e.batch_run(graphs, 1e-6)
    else:
        with lvb200.Server(1e-6, 1 << 30, lanes=1, rule=rule, gain=gain) as s:
            tickets = [s.submit(g) for g in graphs]
            done = s.drain()
        parts = [done[t].assignment for t in tickets]
        q = [done[t].modularity for t in tickets]
        levels = [done[t].levels for t in tickets]
    for i, c in enumerate(csrs):
        orc = _oracle(c, rule, gain)
        assert np.array_equal(parts[i], orc.assignment), i
        assert levels[i] == len(orc.levels)
        assert abs(q[i] - orc.q) < 1e-9


@pytest.mark.parametrize("name", sorted(GRAPHS))
@pytest.mark.parametrize("rule,gain", [("py", "fp32"), ("cuda", "fp32"), ("py", "fp64")])
def test_single_graph_equals_oracle(name, rule, gain):
    c = GRAPHS[name]()
    with lvb200.Engine(rule=rule, gain=gain) as e:
        res = e.run(lvb200.Graph.from_csr(*c), 1e-6)
    orc = _oracle(c, rule, gain)
    assert [l["passes"] for l in res.levels] == [l.passes for l in orc.levels]
    assert np.array_equal(res.assignment, orc.assignment)
    assert abs(res.modularity - orc.q) < 1e-9
