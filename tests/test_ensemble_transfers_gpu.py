"""Populations of a batched ensemble on their way to the device and back: every run's rows are moved in 16-byte
pieces and a byte tail by one launch, so sizes around a piece, a thread's four pieces and a block's are taken."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("x", "y", "z", "fx", "fy", "fz")


@pytest.mark.parametrize("sizes", [[1], [3, 0, 5], [4, 127, 128, 129], [1023, 1024, 1025, 1, 4095, 4097],
                                   [70001, 2] + [7] * 30])
@pytest.mark.parametrize("ids", [True, False])
def test_runs_without_steps_return_their_populations(sizes, ids):
    from flamegpu2_gb300 import sim, synth
    ens = sim.Ensemble("boids_spatial3d", synth.boids_params(dict(synth.BOIDS_SMALL)))
    rng = np.random.default_rng(5)
    pops = []
    for n in sizes:
        pop = {k: rng.standard_normal(n).astype(np.float32) for k in NAMES}
        if ids:
            pop["_id"] = rng.permutation(n).astype(np.uint32) + 1
        pops.append(pop)
        ens.add_run(0, 1, "Boid", n, pop)
    for _ in range(2):  # the second call moves to and from other memory
        assert ens.simulate() == 0 and ens.stats()["batched"]
        for r, (n, pop) in enumerate(zip(sizes, pops)):
            assert ens.count(r, "Boid") == n
            for k in NAMES:
                np.testing.assert_array_equal(ens.get(r, "Boid", k, np.float32), pop[k])
            want = pop["_id"] if ids else np.arange(1, n + 1, dtype=np.uint32)
            np.testing.assert_array_equal(ens.get(r, "Boid", "_id", np.uint32), want)
    ens.close()


def test_an_ensemble_gives_its_memory_back():
    import torch
    from flamegpu2_gb300 import sim, synth
    params = synth.boids_params(dict(synth.BOIDS_SMALL))
    s = sim.Simulation("boids_spatial3d", params)  # simulations keep freed blocks in their pool
    s.set_population("Boid", 1000, synth.boids_population(1000, 0.0, 64.0, 1))
    s.step(1)
    s.close()

    def free_after(n):
        ens = sim.Ensemble("boids_spatial3d", params)
        ens.add_run(0, 1, "Boid", n, {k: np.zeros(n, np.float32) for k in NAMES})
        assert ens.simulate() == 0 and ens.stats()["batched"]
        ens.close()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]
    before = free_after(1000)
    assert free_after(4_000_000) >= before - (64 << 20)  # its columns alone are 224 MB
