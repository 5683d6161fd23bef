"""Populations set and read back through page-locked buffers and from device
columns: row counts around the 16-byte pieces of the transfer launch, element
sizes of 4 and 8 bytes, more than eight columns, buffers at an odd address,
and ids left to be assigned in the last partial piece."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODELS = {"Boid": ("boids_spatial3d", {k: ("f4", 1) for k in ("x", "y", "z", "fx", "fy", "fz")}),
          "agent": ("birth_death", {**{f"f{k}": ("f4", 1) for k in range(8)}, "counter": ("i4", 1)}),
          "cell": ("game_of_life", {"pos": ("u4", 2), "is_alive": ("u4", 1)})}


def _columns(agent, n, seed):
    rng = np.random.default_rng(seed)
    cols = {"_id": (rng.permutation(n) + 1).astype(np.uint32)}
    for k, (t, e) in MODELS[agent][1].items():
        cols[k] = rng.integers(0, 60, (n, e) if e > 1 else n).astype(t)
    return cols


def _pinned(a, offset=0):
    import torch
    buf = torch.empty(a.nbytes + 16, dtype=torch.uint8).pin_memory().numpy()[offset:offset + a.nbytes].view(a.dtype).reshape(a.shape)
    buf[...] = a
    return buf


@pytest.mark.parametrize("offset", [0, 4])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1021, 1024])
@pytest.mark.parametrize("agent", MODELS)
def test_pinned_and_device_round_trips(agent, n, offset):
    import torch
    from flamegpu2_gb300 import sim
    s = sim.Simulation(MODELS[agent][0])
    for seed in (1, 2):
        cols = _columns(agent, n, seed)
        s.set_population(agent, n, {k: _pinned(v, offset) for k, v in cols.items()})
        outs = {k: _pinned(np.zeros_like(v), offset) for k, v in cols.items()}
        assert s.get_population(agent, outs) == n
        for k in cols:
            np.testing.assert_array_equal(outs[k], cols[k])
    cols = _columns(agent, n, 3)
    dev = {}
    for k, v in cols.items():
        b = torch.zeros(v.nbytes + 16, dtype=torch.uint8, device="cuda")[offset:offset + v.nbytes]
        b.copy_(torch.from_numpy(np.frombuffer(v.tobytes(), np.uint8).copy()))
        dev[k] = b
    torch.cuda.synchronize()
    s.reset_population_device(agent, n, dev, n + 1)
    assert s.count(agent) == n
    for k, v in cols.items():
        np.testing.assert_array_equal(s.get(agent, k, v.dtype, v.shape[1] if v.ndim > 1 else 1), v)
    s.close()


@pytest.mark.parametrize("n,unset", [(5, 4), (1021, 1020), (1024, 3)])
def test_an_unset_id_in_any_piece_is_assigned(n, unset):
    from flamegpu2_gb300 import sim
    cols = _columns("Boid", n, 7)
    cols["_id"][unset] = 0
    s = sim.Simulation("boids_spatial3d")
    s.set_population("Boid", n, {k: _pinned(v) for k, v in cols.items()})
    ids = s.get("Boid", "_id", np.uint32)
    assert np.all(ids > 0) and len(np.unique(ids)) == n
    np.testing.assert_array_equal(np.delete(ids, unset), np.delete(cols["_id"], unset))
    s.close()


def test_device_population_gives_births_the_next_ids():
    import torch
    from flamegpu2_gb300 import sim
    n = 4097
    cols = _columns("agent", n, 5)
    s = sim.Simulation("birth_death", [0.0, 1.0, 1])
    for next_id in (n + 1, 50_000):
        dev = {k: torch.from_numpy(v.view(np.int32) if v.dtype == np.uint32 else v).cuda() for k, v in cols.items()}
        s.reset_population_device("agent", n, dev, next_id)
        s.step(1)
        ids = s.get("agent", "_id", np.uint32)
        np.testing.assert_array_equal(ids, np.concatenate([cols["_id"], next_id + np.arange(n, dtype=np.uint32)]))
        assert s.agent_steps() > 0
    s.close()


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 4096, 4097, 700_001, 6_000_001])
def test_columns_copied_to_device_tensors(n):
    """Sizes around a piece, a thread's round and a grid's; a tensor at an odd address; part of a column."""
    import torch
    from flamegpu2_gb300 import sim
    s = sim.Simulation("boids_spatial3d")
    cols = _columns("Boid", n, 3)
    s.set_population("Boid", n, cols)
    for k, offset, m in (("x", 0, n), ("fz", 1, n), ("_id", 4, n), ("y", 0, (n + 1) // 2)):
        buf = torch.full((n + 8,), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        s.get_device("Boid", k, buf[offset:offset + m])
        s.synchronize()
        got = buf.cpu().numpy()
        np.testing.assert_array_equal(got[offset:offset + m].view(cols[k].dtype), cols[k][:m])
        assert (got[:offset] == -1).all() and (got[offset + m:] == -1).all()
    s.close()


@pytest.mark.parametrize("n", [5, 100_003])
def test_a_variable_given_twice_keeps_its_last_column(n):
    """The copies go in the order given; the variable that is missing keeps its values."""
    import ctypes as C
    import torch
    from flamegpu2_gb300 import sim
    s = sim.Simulation("boids_spatial3d")
    before, after = _columns("Boid", n, 11), _columns("Boid", n, 12)
    s.set_population("Boid", n, before)
    names = ["_id", "x", "y", "z", "fx", "fy", "x"]
    cols = [torch.from_numpy(after[k].view(np.int32)).cuda() for k in names]
    cols[1].fill_(0)  # the first x
    torch.cuda.synchronize()
    rc = sim.core().fgs_reset_population_device(
        s._h, b"Boid", b"default", n, len(names), (C.c_char_p * len(names))(*[k.encode() for k in names]),
        (C.c_void_p * len(names))(*[c.data_ptr() for c in cols]), n + 2)
    assert rc == 0 and s.count("Boid") == n
    for k in ("x", "y", "z", "fx", "fy"):
        np.testing.assert_array_equal(s.get("Boid", k, np.float32), after[k])
    np.testing.assert_array_equal(s.get("Boid", "fz", np.float32), before["fz"])
    s.close()
