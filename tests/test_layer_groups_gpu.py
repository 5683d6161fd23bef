"""Functions of one layer side by side and one after another: every column of every list equal, bit for bit, over steps
in which lists outgrow their buffers. The layers hold functions that touch nothing in common and every kind that does:
two readers of one spatial list (it is built, and their agents are sorted by it), a list written and read in one layer,
births into another type, a birth that joins two earlier groups, transitions both ways, deaths, a brute-force list read
by two (which need not wait for each other), and a macro property updated by two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LISTS = [("A", "default"), ("B", "default"), ("C", "default"), ("D", "idle"), ("D", "busy")]
COLUMNS = {"_id": np.uint32, "x": np.float32, "y": np.float32, "v": np.uint32, "s": np.float32}


def _run(n, macro, concurrent, graphs, steps):
    from flamegpu2_gb300 import sim
    s = sim.Simulation("layer_groups", [macro])
    s.set_config("inLayerConcurrency", concurrent)
    s.configure(steps=1, seed=5, use_graphs=graphs)
    rng = np.random.default_rng(n)
    for agent, state in LISTS[:4]:
        s.set_population(agent, n, {"x": rng.uniform(0, 30, n).astype(np.float32), "y": rng.uniform(0, 30, n).astype(np.float32),
                                    "v": rng.integers(0, 1 << 32, n, dtype=np.uint32), "s": np.zeros(n, np.float32)}, state=state)
    out, counts = [], []
    for k in steps:
        s.step(k)
        counts.append([s.count(a, st) for a, st in LISTS])
        out += [s.get(a, c, t, state=st) for a, st in LISTS for c, t in COLUMNS.items()]
    s.close()
    return counts, out


@pytest.mark.parametrize("macro", [0, 1])
@pytest.mark.parametrize("n", [1, 900, 6000])
def test_concurrent_and_sequential_layers_agree(n, macro):
    steps = (1, 1, 6, 7)
    counts, expect = _run(n, macro, False, False, steps)
    if n >= 900:
        first, last = np.array(counts[0]), np.array(counts[-1])
        assert (first > 0).all() and last[2] > 1.5 * n  # C outgrows the room for n and for 1,024
        assert len({tuple(c) for c in counts}) == len(counts)
    for concurrent, graphs in ((False, True), (True, False), (True, True), (True, True)):
        c, got = _run(n, macro, concurrent, graphs, steps)
        assert c == counts
        for a, b in zip(got, expect):
            np.testing.assert_array_equal(a, b)
