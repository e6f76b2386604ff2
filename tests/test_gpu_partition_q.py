"""Modularity of a given partition (lv_modularity_fp64) over rows of every
length its sweep treats apart: empty, short, above 256 entries (listed in
chunks of 4,096 that all blocks share) and more chunks than the list holds;
partitions of one community, of many and of more than a block's cache of
1,024 totals holds.
Reference: the same sums in numpy, FP64.  The FP32 weights' FP64 sums are
exact; only the squared totals round (n terms, each to 2^-53 of a sum that is
at most 1 after the division), so 1e-12 is far above the difference."""
import numpy as np
import pytest

import lvb200

pytestmark = pytest.mark.gpu


def _csr(degrees, seed):
    rng = np.random.default_rng(seed)
    n = len(degrees)
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(degrees)
    col = rng.integers(0, n, int(off[-1])).astype(np.uint32)
    return n, off, col, rng.uniform(0.1, 2.0, len(col)).astype(np.float32)


def _q(n, off, col, w, part):
    row = np.repeat(part, np.diff(off.astype(np.int64)))
    w = w.astype(np.float64)
    tot = np.bincount(row, weights=w, minlength=n)
    m2 = w.sum()
    return w[row == part[col]].sum() / m2 - np.square(tot / m2).sum()


@pytest.mark.parametrize("degrees", [
    [3], [0, 0, 5, 0], [1] * 31, [2] * 33, [255, 256, 257, 8], [1024] * 4, [6] * 9000, [1025, 1, 0, 4096, 4097, 9000] * 7,
    [60_000, 50_000, 7], [0] * 300 + [13] * 700 + [2000]])
def test_q_of_partition_equals_numpy(degrees):
    n, off, col, w = _csr(degrees, seed=len(degrees))
    rng = np.random.default_rng(7)
    with lvb200.Engine() as e:
        e.load(lvb200.Graph.from_csr(n, off, col, w))
        for parts in (1, max(1, n // 3), n):
            part = rng.integers(0, parts, n).astype(np.uint32)
            assert abs(e.modularity(part) - _q(n, off, col, w, part)) < 1e-12


def test_partition_id_out_of_range_is_refused():
    n, off, col, w = _csr([5] * 1000, seed=1)
    part = np.zeros(n, np.uint32)
    with lvb200.Engine() as e:
        e.load(lvb200.Graph.from_csr(n, off, col, w))
        good = e.modularity(part)
        for bad in (n, 0xFFFFFFFF):
            part[777] = bad
            with pytest.raises(lvb200.LouvainError) as err:
                e.modularity(part)
            assert err.value.status == 1
        part[777] = 0
        assert e.modularity(part) == good
