"""The multi-block merge sums a large community's first neighbours in shared
memory (communities of at least 2^18 entries) and adds the rest as they come:
the contracted rows of a given partition with communities on both sides of
that size, whole and fractional weights, equal the oracle's."""
import numpy as np
import pytest

import lvb200
import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 0.25])
def test_large_communities(scale):
    rng = np.random.default_rng(3)
    n, m = 60000, 900000
    a, b = rng.integers(0, n, m), rng.integers(0, n, m)
    e = np.unique(np.minimum(a, b)[a != b] * n + np.maximum(a, b)[a != b])
    a, b = e // n, e % n
    w = (rng.integers(1, 5, len(e)) * scale).astype(np.float32)
    s, d, w = np.r_[a, b], np.r_[b, a], np.r_[w, w]
    o = np.lexsort((d, s))
    s, d, w = s[o], d[o], w[o]
    off = np.searchsorted(s, np.arange(n + 1)).astype(np.uint64)
    # communities: half the vertices, a seventh, 6,000 and singletons
    size = np.r_[n // 2, n // 7, 6000, np.ones(n - n // 2 - n // 7 - 6000, int)]
    comm = np.repeat(np.arange(len(size)), size)[rng.permutation(n)]
    first = np.full(len(size), n)
    np.minimum.at(first, comm, np.arange(n))
    comm = first[comm]  # an id of the community's own vertices
    g = pyoracle.CSR(n, off, d.astype(np.uint32), w.astype(np.float64))
    with lvb200.Engine() as eng:
        eng.load(lvb200.Graph.from_csr(n, off, d.astype(np.uint32), w))
        eng.set_level_comm(comm.astype(np.uint32))
        eng.phase_aggregate()
        n2, off2, col2, w2 = eng.level_csr()
    o2, _ = pyoracle.contract(g, comm.astype(np.uint32), rows="sorted", prec="fp32")
    assert n2 == o2.n and np.array_equal(off2, o2.off)
    row = np.repeat(np.arange(n2), np.diff(off2).astype(np.int64))
    k = np.lexsort((col2, row))
    assert np.array_equal(col2[k], o2.col)
    assert np.array_equal(w2[k].astype(np.float64), o2.w)
