"""Birth/death compaction at the edges of its tiles (1,024 rows), of its
look-back (128 tiles a round) and of one block's births (256 at a time),
through the C ABI against numpy, every value exactly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# element types of one row: groups of four columns with and without an odd width, the id last
LAYOUTS = {"words": ["f4"] * 5, "mixed": ["f4", "f8", "u1", "f4", "f4", "3f4", "f4", "i4", "f4"], "id": []}


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("n,p_born,room", [(1023, 0.3, None), (1024, 1.0, None), (1025, 0.0, None), (2048, 0.7, None),
                                           (131_072, 0.2, None), (131_073, 0.2, None), (300_000, 0.6, 50)])
def test_compaction_tiles(n, p_born, room, layout):
    import torch
    from flamegpu2_gb300 import capi
    L = capi.lib()
    rng = np.random.default_rng(n)
    alive = (rng.random(n) < 0.7).astype(np.int32)
    born = ((rng.random(n) < p_born) & (alive == 1)).astype(np.int32)
    born[rng.random(n) < 0.1] *= 2  # claimed ids: the staging row's is kept
    surv, kids = np.nonzero(alive)[0], np.nonzero(born)[0]
    total = len(surv) + len(kids)
    cap = total + 3 if room is None else total - room
    rows, births, outs = [], [], []
    for t in LAYOUTS[layout] + ["i4"]:
        per = np.dtype(t).itemsize
        rows.append(rng.integers(0, 256, (n, per), dtype=np.uint8))
        births.append(rng.integers(0, 256, (n, per), dtype=np.uint8))
        outs.append(torch.zeros((cap, per), dtype=torch.uint8, device="cuda"))
    gpu = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    ins, bins = [gpu(r) for r in rows], [gpu(b) for b in births]
    ncols = len(ins)
    d_n, n_out = torch.tensor([n], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    next_id = torch.tensor([7], dtype=torch.int32, device="cuda")
    a_t, b_t = gpu(alive), gpu(born)
    ws = capi.Workspace(L.fg_compact_workspace_size(n))
    for _ in range(2):  # the second call uses the other tile statuses
        next_id.fill_(7)
        capi.check(L.fg_compact_agents(n, d_n.data_ptr(), a_t.data_ptr(), b_t.data_ptr(), capi.columns(list(zip(ins, outs))),
                                       capi.columns(list(zip(bins, outs))), ncols, ncols - 1, next_id.data_ptr(), None,
                                       n_out.data_ptr(), cap, ws.ptr, ws.nbytes, capi.stream_handle()), "fg_compact_agents")
    torch.cuda.synchronize()
    assert ws.status() == (0 if room is None else capi.FG_ERR_CAPACITY)
    assert int(n_out.item()) == min(total, cap) and int(next_id.item()) == 7 + len(kids)
    ids = (7 + np.arange(len(kids))).astype(np.int32)
    kept = born[kids] == 2
    for c in range(ncols):
        kid = births[c][kids].copy()
        if c == ncols - 1:
            kid[~kept] = ids[~kept].view(np.uint8).reshape(-1, 4)
        np.testing.assert_array_equal(outs[c].cpu().numpy()[:total], np.concatenate([rows[c][surv], kid])[:cap])


@pytest.mark.parametrize("n,spare", [(1, 1), (1024, 1), (5_000, 3), (5_000, 600), (100_000, 90)])
def test_population_tiles_below_its_capacity(n, spare):
    """Calls in a row on one workspace, as a simulation makes them (the count in place, both status arrays in turn),
    with blocks past the population's tiles: they read the count and the parity that the last block then changes."""
    import torch
    from flamegpu2_gb300 import capi
    L = capi.lib()
    cap = n + spare * 1024
    rng = np.random.default_rng(n + spare)
    value = np.arange(n, dtype=np.int32)
    cols = [torch.zeros(cap, dtype=torch.int32, device="cuda") for _ in range(2)]
    cols[0][:n] = torch.from_numpy(value).cuda()
    births = torch.full((cap,), -7, dtype=torch.int32, device="cuda")
    d_n = torch.tensor([n], dtype=torch.int32, device="cuda")
    ws = capi.Workspace(L.fg_compact_workspace_size(cap))
    flags, expect = [], value
    for _ in range(24):
        alive, born = (rng.random(cap) < 0.9).astype(np.int32), (rng.random(cap) < 0.1).astype(np.int32)
        m = len(expect)
        expect = np.concatenate([expect[alive[:m] == 1], np.full(born[:m].sum(), -7, np.int32)])
        flags.append((torch.from_numpy(alive).cuda(), torch.from_numpy(born).cuda()))
        assert len(expect) <= cap
    torch.cuda.synchronize()
    for k, (alive, born) in enumerate(flags):  # nothing waits between the calls
        a, b = cols[k % 2], cols[1 - k % 2]
        capi.check(L.fg_compact_agents(cap, d_n.data_ptr(), alive.data_ptr(), born.data_ptr(), capi.columns([(a, b)]),
                                       capi.columns([(births, b)]), 1, -1, None, None, d_n.data_ptr(), cap, ws.ptr,
                                       ws.nbytes, capi.stream_handle()), "fg_compact_agents")
    torch.cuda.synchronize()
    assert ws.status() == 0
    assert int(d_n.item()) == len(expect)
    np.testing.assert_array_equal(cols[0].cpu().numpy()[:len(expect)], expect)
