"""The union's modularity sweep cuts every moving graph's entries into chunks
of 4,096: graphs whose entry counts lie around a chunk's end, graphs without
edges at the union's start, middle and end, and many graphs in one chunk's
reach give what a run of each graph alone gives (partitions, levels; Q to the
order of its FP64 sums, 1e-12)."""
import numpy as np
import pytest

import lvb200

pytestmark = pytest.mark.gpu


def _regular(n, degree, seed):
    rng = np.random.default_rng(seed)
    src = np.repeat(np.arange(n), degree)
    dst = np.where(rng.random(len(src)) < 0.7, (src + rng.integers(0, 9, len(src))) % n,
                   rng.integers(0, n, len(src)))
    return lvb200.Graph.from_csr(n, np.arange(n + 1) * degree, dst,
                                 rng.uniform(0.5, 1.5, len(src)))


SHAPES = [(7, 0), (1024, 4), (1365, 3), (4097, 1), (1, 1), (1, 0), (2048, 4), (3, 2), (8191, 1),
          (4096, 3), (700, 40), (5, 0)]


@pytest.mark.parametrize("order", ["as_is", "reversed", "shuffled_with_tiny"])
@pytest.mark.parametrize("use_graphs", [True, False])
def test_union_equals_lone_runs(order, use_graphs):
    shapes = list(SHAPES)
    if order == "reversed":
        shapes.reverse()
    elif order == "shuffled_with_tiny":
        rng = np.random.default_rng(3)
        shapes = shapes + [(int(n), int(d)) for n, d in zip(rng.integers(1, 30, 1500),
                                                            rng.integers(0, 6, 1500))]
        shapes = [shapes[i] for i in rng.permutation(len(shapes))]
    graphs = [_regular(n, d, seed=i) for i, (n, d) in enumerate(shapes)]
    with lvb200.Engine(use_graphs=use_graphs) as e:
        for _ in range(2):
            parts, q, levels, _ = e.batch_run(graphs, 1e-6)
    with lvb200.Engine() as e:
        for i in list(range(0, len(graphs), max(1, len(graphs) // 60))):
            alone = e.run(graphs[i], 1e-6)
            assert np.array_equal(parts[i], alone.assignment), shapes[i]
            assert levels[i] == len(alone.levels)
            assert abs(q[i] - alone.modularity) < 1e-12
