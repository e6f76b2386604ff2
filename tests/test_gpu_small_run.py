"""The small-run kernel (every remaining level of a small graph in one
launch) against the level-by-level path, which use_graphs=False selects and
which the parity tests pin to the oracle: identical partitions, levels,
passes and entry counts, Q to the order of its FP64 sums (1e-12), at the
edges of what the kernel takes -- vertices and entries around its limits,
rows too long for it, rows of every bucket, no edges, one vertex -- under
both rules and both gain modes, and through the phase calls."""
import numpy as np
import pytest

import lvb200
import lvgen

pytestmark = pytest.mark.gpu


def _graph(name):
    rng = np.random.default_rng(len(name))
    if name == "one_vertex":
        return lvb200.Graph.from_edges(1, [0], [0], [2.0])
    if name == "no_edges":
        return lvb200.Graph.from_edges(50, [], [], [])
    if name == "zero_weights":
        return lvb200.Graph.from_edges(4, [0, 1], [1, 2], [0.0, 0.0])
    if name == "star1000":
        return lvb200.Graph.from_edges(*lvgen.star(1000))
    if name == "star3000":  # a row above 2,048 entries
        return lvb200.Graph.from_edges(*lvgen.star(3000))
    if name == "dense":  # every row in the block class
        n = 330
        s, d = np.triu_indices(n, 1)
        return lvb200.Graph.from_edges(n, s, d, rng.uniform(0.1, 1, len(s)))
    if name == "loops_dups":
        s, d = rng.integers(0, 40, 900), rng.integers(0, 40, 900)
        return lvb200.Graph.from_edges(60, s, d, rng.integers(1, 5, 900))
    if name == "chain":  # many levels
        s = np.arange(2047)
        return lvb200.Graph.from_edges(2048, s, s + 1, np.ones(2047))
    kind, n = name.split("_")
    n = int(n)
    if kind == "banded":
        return lvb200.Graph.from_edges(*lvgen.banded_fem(n=n, half_band=30, target_entries=20 * n,
                                                         seed=n))
    if kind == "sbm":
        return lvb200.Graph.from_edges(*lvgen.sbm(n, 8, mean_deg=15.0, seed=n))
    if kind == "rmat":
        return lvb200.Graph.from_edges(*lvgen.rmat(n, edge_factor=12, seed=n, unit=False))
    return lvb200.Graph.from_edges(*lvgen.planted_powerlaw(
        n=n, target_edges=3 * n, max_deg=min(400, n // 8), comm_max=max(20, n // 10), seed=n))


NAMES = ["one_vertex", "no_edges", "zero_weights", "star1000", "star3000", "dense", "loops_dups",
         "chain", "sbm_64", "sbm_130", "banded_1000", "sbm_1024", "sbm_1025", "sbm_2048", "sbm_2049",
         "rmat_9", "rmat_11",
         "planted_500", "planted_20000"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("rule,gain", [("py", "fp32"), ("cuda", "fp32"), ("py", "fp64"),
                                       ("cuda", "fp64")])
def test_small_run_equals_level_path(name, rule, gain):
    g = _graph(name)
    for limits in (dict(), dict(max_levels=2), dict(max_passes=3)):
        with lvb200.Engine(rule=rule, gain=gain, use_graphs=False, **limits) as e:
            a = e.run(g, 1e-6)
            state_a = e.level_state()
        with lvb200.Engine(rule=rule, gain=gain, **limits) as e:
            for _ in range(2):  # the second run on kept buffers
                b = e.run(g, 1e-6)
            state_b = e.level_state()
        keys = ("n_vertices", "n_entries", "passes", "moved")
        assert [[l[k] for k in keys] for l in a.levels] == [[l[k] for k in keys] for l in b.levels]
        assert np.array_equal(a.assignment, b.assignment)
        assert a.n_communities == b.n_communities and a.edges_processed == b.edges_processed
        assert abs(a.modularity - b.modularity) < 1e-12
        for x, y in zip(a.levels, b.levels):
            assert abs(x["q_start"] - y["q_start"]) < 1e-12
            assert abs(x["q_end"] - y["q_end"]) < 1e-12
        for x, y in zip(state_a, state_b):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("name", ["sbm_130", "planted_500", "rmat_11", "star3000"])
def test_phase_calls_equal_level_path(name):
    g = _graph(name)
    seen = []
    for graphs in (False, True):
        with lvb200.Engine(use_graphs=graphs) as e:
            e.load(g)
            steps = []
            for _ in range(30):
                more, q = e.phase_move(1e-6)
                comm, sz, k = e.level_state()
                steps.append((more, round(q, 12), comm.tolist(), sz.tolist(), k.tolist()))
                if not more:
                    break
                # a second call on the same level goes on from its state
                again, q2 = e.phase_move(1e-6)
                steps.append((again, round(q2, 12), e.level_state()[0].tolist()))
                if not again:
                    break
                e.phase_aggregate()
            steps.append(e.assignment().tolist())
            seen.append(steps)
    assert seen[0] == seen[1]


def test_calls_after_a_small_run():
    """Entry points that need the class lists rebuild them around the state."""
    g = _graph("sbm_130")
    with lvb200.Engine() as e:
        e.run(g, 1e-6)
        before = e.level_state()
        q = e.modularity(before[0])
        e.autotune(reps=1)
        after = e.level_state()
        for x, y in zip(before, after):
            assert np.array_equal(x, y)
        assert e.modularity(after[0]) == q
        e.set_level_comm(before[0])
        assert np.array_equal(e.level_state()[0], before[0])
