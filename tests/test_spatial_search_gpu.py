"""Spatial searches where their range words end: ranges longer than a word
holds beside a first index (the walk then steps through the neighbourhood),
searches nested in another of the same agent, and copied ones. Message counts
against numpy, exactly."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _neighbourhood_sums(counts, wrap):
    """Per bin, the sum of `counts` over its Moore neighbourhood."""
    g, dims = counts.shape[0], counts.ndim
    padded = np.pad(counts, 1, mode="wrap" if wrap else "constant")
    out = np.zeros_like(counts)
    for off in itertools.product((0, 1, 2), repeat=dims):
        out += padded[tuple(slice(o, o + g) for o in off)]
    return out


def _bins(pos, g):
    return tuple(np.minimum(np.floor(pos[:, a]).astype(int), g - 1) for a in range(pos.shape[1]))


@pytest.mark.parametrize("wrap", [False, True])
@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("in_bin", [32767, 32768])
def test_ranges_longer_than_a_range_word_holds(dims, wrap, in_bin):
    # 66,000 messages: 17 bits of index leave 15 for a range's length
    from flamegpu2_gb300 import sim
    n, g = 66_000, 8
    rng = np.random.default_rng(in_bin + dims)
    pos = rng.uniform(0.0, g, (n, dims)).astype(np.float32)
    pos[:in_bin] = rng.uniform(0.01, 0.99, (in_bin, dims))  # one heavy bin, at the domain's corner
    rest = pos[in_bin:]
    rest[np.all(rest < 1.0, axis=1)] += np.float32(1.0)
    counts = np.zeros((g,) * dims, np.int64)
    np.add.at(counts, _bins(pos, g), 1)
    assert counts.max() == in_bin
    s = sim.Simulation("spatial_count", [dims, 0, 0, 0, g, g, g, 1.0, int(wrap), 0])
    cols = {"x": pos[:, 0].copy(), "y": pos[:, 1].copy(), "z": pos[:, 2].copy() if dims == 3 else np.zeros(n, np.float32)}
    s.set_population("agent", n, cols)
    s.step(1)
    got = np.stack([s.get("agent", k, np.float32) for k in ("x", "y", "z")[:dims]], 1)
    visited = s.get("agent", "count", np.uint32)
    if wrap:  # the wrapped function counts each message as one of its lattice's or as a bad one
        visited = visited + s.get("agent", "badCount", np.uint32)
    np.testing.assert_array_equal(visited, _neighbourhood_sums(counts, wrap)[_bins(got, g)])
    s.close()


@pytest.mark.parametrize("wrap", [False, True])
@pytest.mark.parametrize("dims,n", [(2, 1), (2, 700), (3, 1500)])
def test_nested_and_copied_searches(dims, n, wrap):
    from flamegpu2_gb300 import sim
    g = 6
    pos = np.random.default_rng(n).uniform(0.0, g, (n, dims)).astype(np.float32)
    counts = np.zeros((g,) * dims, np.int64)
    np.add.at(counts, _bins(pos, g), 1)
    around = _neighbourhood_sums(counts, wrap)
    s = sim.Simulation("spatial_nested", [dims, 0.0, g, 1.0, int(wrap)])
    s.set_population("agent", n, {k: pos[:, a].copy() for a, k in enumerate(("x", "y", "z")[:dims])})
    s.step(2)
    got = _bins(np.stack([s.get("agent", k, np.float32) for k in ("x", "y", "z")[:dims]], 1), g)
    np.testing.assert_array_equal(s.get("agent", "outer", np.uint32), around[got])
    np.testing.assert_array_equal(s.get("agent", "copied", np.uint32), around[got])
    np.testing.assert_array_equal(s.get("agent", "inner", np.uint32), _neighbourhood_sums(counts * around, wrap)[got])
    s.close()


@pytest.mark.parametrize("wrap", [False, True])
@pytest.mark.parametrize("n", [1, 129, 304 * 128, 304 * 128 + 1])
def test_staged_and_unstaged_walks_agree(n, wrap):
    # two blocks of 128 agents a SM are the most that a launch stages windows for
    from flamegpu2_gb300 import sim, synth
    cells = max(4, int(np.ceil(n ** (1.0 / 3.0))))
    cfg = dict(synth.BOIDS_SMALL, n=n, max_pos=2.0 * cells, wrap=int(wrap))
    pop = synth.boids_population(n, 0.0, 2.0 * cells, 9)
    got = []
    for stage in (96 * 1024, 0):
        s = sim.Simulation("boids_spatial3d", synth.boids_params(cfg))
        s.set_stage_bytes(stage)
        s.set_population("Boid", n, pop)
        s.step(3)
        got.append([s.get("Boid", "_id", np.uint32)] + [s.get("Boid", k, np.float32) for k in ("x", "y", "z", "fx", "fy", "fz")])
        s.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("wrap", [False, True])
@pytest.mark.parametrize("dims,n", [(2, 1), (2, 700), (3, 1500)])
def test_searches_of_a_copied_input_list(dims, n, wrap):
    from flamegpu2_gb300 import sim
    g = 6
    pos = np.random.default_rng(n + 1).uniform(0.0, g, (n, dims)).astype(np.float32)
    counts = np.zeros((g,) * dims, np.int64)
    np.add.at(counts, _bins(pos, g), 1)
    around = _neighbourhood_sums(counts, wrap)
    s = sim.Simulation("spatial_nested", [dims, 0.0, g, 1.0, int(wrap)])
    s.set_population("agent", n, {k: pos[:, a].copy() for a, k in enumerate(("x", "y", "z")[:dims])})
    s.step(1)
    got = _bins(np.stack([s.get("agent", k, np.float32) for k in ("x", "y", "z")[:dims]], 1), g)
    np.testing.assert_array_equal(s.get("agent", "list_outer", np.uint32), around[got])
    pairs = _neighbourhood_sums(counts * around, wrap)[got]
    np.testing.assert_array_equal(s.get("agent", "list_inner", np.uint32), pairs)
    np.testing.assert_array_equal(s.get("agent", "list_swapped", np.uint32), pairs)
    s.close()


@pytest.mark.parametrize("wrap", [False, True])
@pytest.mark.parametrize("g", [1, 2, 3])
@pytest.mark.parametrize("dims", [2, 3])
def test_nested_and_copied_searches_on_small_grids(dims, g, wrap):
    """A grid of one to three bins an axis: the neighbours on both sides of a bin turn round, or are one bin."""
    from flamegpu2_gb300 import sim
    n = 90
    pos = np.random.default_rng(10 * dims + g).uniform(0.0, g, (n, dims)).astype(np.float32)
    counts = np.zeros((g,) * dims, np.int64)
    np.add.at(counts, _bins(pos, g), 1)
    around = _neighbourhood_sums(counts, wrap)
    s = sim.Simulation("spatial_nested", [dims, 0.0, g, 1.0, int(wrap)])
    s.set_population("agent", n, {k: pos[:, a].copy() for a, k in enumerate(("x", "y", "z")[:dims])})
    s.step(1)
    got = _bins(np.stack([s.get("agent", k, np.float32) for k in ("x", "y", "z")[:dims]], 1), g)
    pairs = _neighbourhood_sums(counts * around, wrap)[got]
    for name in ("outer", "copied", "list_outer"):
        np.testing.assert_array_equal(s.get("agent", name, np.uint32), around[got])
    for name in ("inner", "list_inner", "list_swapped"):
        np.testing.assert_array_equal(s.get("agent", name, np.uint32), pairs)
    s.close()
