"""A device with little free memory: runs that need room for one tile's sweep
outputs only must not fail for want of room for several."""
import numpy as np
import pytest

from lsim_b200 import Simulator, gen

pytestmark = pytest.mark.gpu


def test_a_full_device_runs_one_tile_at_a_time():
    torch = pytest.importorskip("torch")
    tiles = 700
    w = gen.generate(n_gates=1500, n_pi=16, n_po=16, n_levels=30, n_patterns=64, seed=4)
    rng = np.random.default_rng(0)
    words = rng.integers(0, 1 << 64, (tiles * 32, 16), dtype=np.uint64)

    def run():
        sim = Simulator(0)
        sim.load_circuit(w["ckt"])
        sim.set_fault_text(w["flst"])
        sim.set_patterns(words, tiles * 2048)
        sim.run()
        return sim, sim.results().copy(), sim.stats()["device_bytes"]

    sim, want, most = run()
    good = sim.good_values(31)
    values = tiles * sim.info().num_elements * 256  # good values of all tiles
    room = values + (64 << 20)
    assert most > values + (256 << 20)  # the sweep outputs of several tiles
    del sim
    free, _ = torch.cuda.mem_get_info(0)
    assert free > room + (64 << 20)
    fill = torch.empty(free - room, dtype=torch.uint8, device="cuda:0")
    try:
        for _ in range(2):
            sim, got, used = run()
            assert np.array_equal(got, want)
            assert used < room
            assert np.array_equal(sim.good_values(31), good)
            sim.run()
            assert np.array_equal(sim.results(), want)
            del sim
    finally:
        del fill
        torch.cuda.empty_cache()
