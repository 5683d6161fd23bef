"""Message builds over rows: populations around one and four grid widths of the
key kernel (4 rows a thread in flight), records of 4, 8 and 12 words, rows in
no order and drifted from bin order, optional rows. Records and PBM exactly
against numpy's stable order."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("optional", [False, True])
@pytest.mark.parametrize("drifted", [False, True])
@pytest.mark.parametrize("n,words", [(255, 1), (311_295, 5), (311_297, 1), (1_245_185, 8)])
def test_build_rows(n, words, drifted, optional):
    import torch
    from flamegpu2_gb300 import capi
    L = capi.lib()
    rng = np.random.default_rng(n + words)
    cells = max(2, int((n / 3.0) ** (1.0 / 3.0)))
    pos = rng.uniform(0.0, cells, (n, 3)).astype(np.float32)
    key_of = lambda p: ((p[:, 2].astype(np.int64) * cells) + p[:, 1].astype(np.int64)) * cells + p[:, 0].astype(np.int64)  # noqa: E731
    if drifted:
        pos = pos[np.argsort(key_of(pos), kind="stable")]
        pos = np.clip(pos + rng.normal(0.0, 0.05, pos.shape), 0.0, np.nextafter(np.float32(cells), np.float32(0))).astype(np.float32)
    key = key_of(pos)
    payload = rng.integers(0, 1 << 30, (n, words)).astype(np.int32)
    valid = (rng.random(n) < 0.8).astype(np.int32) if optional else None
    cols = [torch.from_numpy(np.ascontiguousarray(pos[:, a])).cuda() for a in range(3)] + [torch.from_numpy(payload).cuda()]
    v_t = None if valid is None else torch.from_numpy(valid).cuda()
    g = capi.grid(3, (0, 0, 0), (cells,) * 3, 1.0)
    rec = capi.record_desc(cols)
    out = torch.zeros((n, rec.words), dtype=torch.int32, device="cuda")
    pbm = torch.zeros(g.binCount + 1, dtype=torch.int32, device="cuda")
    ws = capi.Workspace(L.fg_spatial_build_workspace_size(n, g.binCount))
    for _ in range(2):
        capi.check(L.fg_spatial_build(C.byref(g), n, None, cols[0].data_ptr(), cols[1].data_ptr(), cols[2].data_ptr(),
                                      capi.ptr(v_t), C.byref(rec), out.data_ptr(), pbm.data_ptr(), ws.ptr, ws.nbytes,
                                      capi.stream_handle()), "fg_spatial_build")
    torch.cuda.synchronize()
    keep = np.arange(n) if valid is None else np.nonzero(valid)[0]
    order = keep[np.argsort(key[keep], kind="stable")]
    counts = np.bincount(key[keep], minlength=cells ** 3)
    np.testing.assert_array_equal(pbm.cpu().numpy(), np.concatenate([[0], np.cumsum(counts)]))
    got = out.cpu().numpy()[:len(order)]
    np.testing.assert_array_equal(got[:, :3].view(np.float32), pos[order])
    np.testing.assert_array_equal(got[:, 3:3 + words], payload[order])
    assert ws.status() == 0


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("cells", [1, 6, 7, 16])  # 216 and 343 bins: at and past the buckets that share by match
def test_key_groups_in_a_model_and_standalone(cells, shuffled):
    # a population whose warps hold long runs, single lanes and messages not output
    from flamegpu2_gb300 import sim
    n, rng = 5003, np.random.default_rng(cells)
    pos = rng.uniform(0.0, cells, (n, 3)).astype(np.float32)
    if not shuffled:
        key = (pos[:, 2].astype(int) * cells + pos[:, 1].astype(int)) * cells + pos[:, 0].astype(int)
        pos = pos[np.argsort(key, kind="stable")]
    out = (rng.random(n) < 0.7).astype(np.int32)
    s = sim.Simulation("spatial_count", [3, 0, 0, 0, cells, cells, cells, 1.0, 0, 1])
    s.set_population("agent", n, {"x": pos[:, 0].copy(), "y": pos[:, 1].copy(), "z": pos[:, 2].copy(), "do_output": out})
    s.step(2)
    got = np.stack([s.get("agent", k, np.float32) for k in ("x", "y", "z")], 1)
    counts = np.zeros((cells,) * 3, np.int64)
    np.add.at(counts, tuple(pos[out == 1].astype(int).T), 1)
    padded = np.pad(counts, 1)
    around = sum(padded[a:a + cells, b:b + cells, c:c + cells] for a in range(3) for b in range(3) for c in range(3))
    np.testing.assert_array_equal(s.get("agent", "count", np.uint32), around[tuple(got.astype(int).T)])
    s.close()
