"""The G-lane move kernels' grouping of equal neighbour communities (16 and
32 lanes: slots in shared memory, 4 and 8: shuffles) on rows of every length
around a group's, from all-distinct communities (a level's first pass) to
all-equal ones (its last): runs equal the oracle's.  Integer weights, so every
sum is exact and the partitions are equal, whatever the order."""
import numpy as np
import pytest

import lvb200
import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [1, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33])
@pytest.mark.parametrize("use_graphs", [True, False])
def test_regular_rows(degree, use_graphs):
    rng = np.random.default_rng(degree)
    n = 1501  # ids spread over blocks: the last group and warp are partial
    src = np.repeat(np.arange(n), degree)
    near = (src + rng.integers(1, 12, len(src))) % n
    dst = np.where(rng.random(len(src)) < 0.8, near, rng.integers(0, n, len(src)))
    w = rng.integers(1, 4, len(src)).astype(np.float32)
    # directed rows of exactly `degree` entries: what the kernels see
    off = np.arange(n + 1, dtype=np.uint64) * degree
    g = lvb200.Graph.from_csr(n, off, dst, w)
    orc = pyoracle.louvain(pyoracle.CSR(n, off, dst.astype(np.uint32), w.astype(np.float64)), 1e-6,
                           rule="py", prec="fp32", rows="sorted")
    with lvb200.Engine(use_graphs=use_graphs) as e:
        res = e.run(g, 1e-6)
    assert [l["passes"] for l in res.levels] == [l.passes for l in orc.levels]
    assert np.array_equal(res.assignment, orc.assignment)
    assert abs(res.modularity - orc.q) < 1e-9
