"""Agent sorts whose columns move one after another by the stable permutation
(more column bytes than L2 holds, rows in no order) and at once (drifted, in
order, or half of each), through the C ABI against numpy's stable order."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["random", "half", "drifted", "sorted", "long"])
@pytest.mark.parametrize("n", [5000, 2_500_000])
def test_sort_moves_every_column(n, order):
    import torch
    from flamegpu2_gb300 import capi
    L = capi.lib()
    rng = np.random.default_rng(n + len(order))
    cells = 8 if order == "long" else max(2, int((n / 3.0) ** (1.0 / 3.0)))
    pos = rng.uniform(0.0, cells, (n, 3)).astype(np.float32)
    w = np.float32(cells)
    cell = lambda p, a: np.floor((p[:, a] / w) * w).astype(np.int64)  # noqa: E731  (the sort key's own float32 arithmetic)
    key_of = lambda p: (cell(p, 2) * cells + cell(p, 1)) * cells + cell(p, 0)  # noqa: E731
    if order in ("half", "drifted", "sorted"):
        pos = pos[np.argsort(key_of(pos), kind="stable")]
    if order == "drifted":
        top = np.nextafter(np.float32(cells), np.float32(0))
        pos = np.clip(pos + rng.normal(0.0, 0.05, pos.shape), 0.0, top).astype(np.float32)
    if order == "half":
        pos[:n // 2] = rng.permutation(pos[:n // 2])
    cols = [np.ascontiguousarray(pos[:, a]) for a in range(3)]
    cols += [rng.integers(0, 1 << 30, n).astype(np.int32) for _ in range(7)]  # ten 4-byte columns
    cols += [rng.integers(0, 1 << 60, n) for _ in range(3)]                   # three 8-byte ones
    cols += [rng.integers(0, 250, n).astype(np.uint8), rng.integers(0, 250, n).astype(np.int16),
             rng.integers(0, 250, (n, 4)).astype(np.int32), rng.integers(0, 250, (n, 3)).astype(np.int32)]
    ins = [torch.from_numpy(c).cuda() for c in cols]
    outs = [torch.zeros_like(c) for c in ins]
    mixed = rng.permutation(len(ins))  # the order they are given in is free
    g = capi.grid(3, (0, 0, 0), (cells,) * 3, 1.0)
    perm = torch.zeros(n, dtype=torch.int32, device="cuda")
    ws = capi.Workspace(L.fg_spatial_sort_workspace_size(n, C.byref(g)))
    table = capi.columns([(ins[k], outs[k]) for k in mixed])
    expect = np.argsort(key_of(pos), kind="stable")
    for perm_out in (None, perm):
        for o in outs:
            o.zero_()
        capi.check(L.fg_spatial_sort_agents(C.byref(g), n, None, ins[0].data_ptr(), ins[1].data_ptr(), ins[2].data_ptr(), table,
                                            len(ins), capi.ptr(perm_out), ws.ptr, ws.nbytes, capi.stream_handle()),
                   "fg_spatial_sort_agents")
        torch.cuda.synchronize()
        for c, o in zip(cols, outs):
            np.testing.assert_array_equal(o.cpu().numpy(), c[expect])
    np.testing.assert_array_equal(perm.cpu().numpy(), expect)
    assert ws.status() == 0


@pytest.mark.parametrize("n", [1, 33, 8_191, 20_000, 100_001, 400_031])
def test_rows_placed_far_apart_are_counted(n):
    """What decides how the columns move: rows more than 4,096 places from the row before them in their 32, counted by
    the placement (the third word of the workspace's header) at ragged ends too. One row a bin, so places are known."""
    import torch
    from flamegpu2_gb300 import capi
    L = capi.lib()
    room = 1_700_000  # of eight 8-byte columns: more than L2 holds
    gx, gy = 1024, room // 1024 + 1
    place = np.random.default_rng(n).permutation(n)
    x, y = torch.zeros(room, device="cuda"), torch.zeros(room, device="cuda")
    x[:n] = torch.from_numpy((place % gx + 0.5).astype(np.float32)).cuda()
    y[:n] = torch.from_numpy((place // gx + 0.5).astype(np.float32)).cuda()
    wide = [torch.arange(room, device="cuda") + (k << 40) for k in range(8)]
    outs = [torch.zeros_like(c) for c in wide]
    g = capi.grid(2, (0, 0), (gx, gy), 1.0)
    d_n = torch.tensor([n], dtype=torch.int32, device="cuda")
    ws = capi.Workspace(L.fg_spatial_sort_workspace_size(room, C.byref(g)))
    capi.check(L.fg_spatial_sort_agents(C.byref(g), room, d_n.data_ptr(), x.data_ptr(), y.data_ptr(), None,
                                        capi.columns(list(zip(wide, outs))), 8, None, ws.ptr, ws.nbytes,
                                        capi.stream_handle()), "fg_spatial_sort_agents")
    torch.cuda.synchronize()
    far = (np.abs(np.diff(place)) > 4096) & (np.arange(1, n) % 32 != 0)
    assert int(ws.buf.view(torch.int32)[2]) == far.sum()
    for k, o in enumerate(outs):
        np.testing.assert_array_equal(o[:n].cpu().numpy(), np.argsort(place) + (k << 40))
    assert ws.status() == 0


def test_kernels_of_a_step_count_the_column_gather():
    """28-byte agents: 96 MB of columns are 3,595,117 agents and a part; above, the sort has one kernel more."""
    import torch
    from flamegpu2_gb300 import sim
    kernels = []
    for n in (3_595_117, 3_595_118):
        s = sim.Simulation("spatial_payload", [2, 0.0, 1896.0, 4.0])
        cols = {k: torch.rand(n, device="cuda") * 1896.0 for k in ("x", "y", "p0", "p1", "p2", "p3")}
        cols["_id"] = torch.arange(1, n + 1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        s.reset_population_device("agent", n, cols, n + 1)
        s.step(1)
        s.synchronize()
        kernels.append(s.stats()["kernels_per_step"])
        s.close()
    assert kernels[1] == kernels[0] + 1
