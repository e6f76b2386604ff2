"""Tables of the move and merge kernels on levels of whole weights (32-bit
sums) and of others (FP64 sums): rows of every table's edge lengths, whole
weights, whole weights whose total passes the 32-bit limit, and quarters.
Every sum is exact, so partitions equal the oracle's."""
import numpy as np
import pytest

import lvb200
import pyoracle

pytestmark = pytest.mark.gpu


def graph(scale, seed):
    # hubs of the degrees at which rows change kernels, over small cliques
    rng = np.random.default_rng(seed)
    n, size = 6000, 12
    v = np.arange(n)
    src = [np.repeat(v, size - 1)]
    dst = [(v // size * size)[:, None] + (v[:, None] + np.arange(1, size)) % size]
    for hub, d in enumerate((33, 84, 85, 127, 128, 319, 320, 512, 2048, 2049, 4096, 5500)):
        src.append(np.full(d, hub * 400))
        dst.append(rng.choice(n, d, replace=False))
    src, dst = np.concatenate(src), np.concatenate([x.ravel() for x in dst])
    keep = src != dst
    e = np.unique(np.minimum(src, dst)[keep] * n + np.maximum(src, dst)[keep])
    a, b = e // n, e % n
    w = (rng.integers(1, 4, len(e)) * scale).astype(np.float32)
    s, d, w = np.r_[a, b], np.r_[b, a], np.r_[w, w]
    o = np.lexsort((d, s))
    off = np.searchsorted(s[o], np.arange(n + 1)).astype(np.uint64)
    return n, off, d[o].astype(np.uint32), w[o]


# 16384: total weight past 2^31; 0.25: fractions
@pytest.mark.parametrize("scale", [1, 3, 16384, 0.25])
@pytest.mark.parametrize("rule,gain", [("py", "fp32"), ("cuda", "fp32"), ("py", "fp64")])
def test_equals_oracle(scale, rule, gain):
    n, off, col, w = graph(scale, 7)
    with lvb200.Engine(rule=rule, gain=gain) as e:
        res = e.run(lvb200.Graph.from_csr(n, off, col, w), 1e-6)
    orc = pyoracle.louvain(pyoracle.CSR(n, off, col, w.astype(np.float64)), 1e-6, rule=rule,
                           prec=gain, rows="sorted")
    assert [l["passes"] for l in res.levels] == [l.passes for l in orc.levels]
    assert np.array_equal(res.assignment, orc.assignment)
    assert abs(res.modularity - orc.q) < 1e-9
