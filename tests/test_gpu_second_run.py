"""A handle's second run costs what its third costs: nothing is set up for
later runs that so few runs cannot earn back."""
import time

import numpy as np
import pytest

from lsim_b200 import Simulator, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gates,patterns", [(400, 64), (2000, 64)])
def test_the_second_run_costs_what_the_third_costs(gates, patterns):
    w = gen.generate(n_gates=gates, n_pi=32, n_po=32, n_levels=20, n_patterns=patterns, seed=1, faults="collapsed")
    ratio = []
    for _ in range(7):
        sim = Simulator(0)
        sim.read_text(w["ckt"], w["flst"], w["ptn"])
        spent, got = [], []
        for _ in range(3):
            t = time.perf_counter()
            sim.run()
            spent.append(time.perf_counter() - t)
            got.append(sim.results().copy())
        assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
        ratio.append(spent[1] / spent[2])
    # the least of seven handles: locking host memory in the second run made it 8 to 17
    assert min(ratio) < 4, ratio


def test_results_through_the_change_of_memory():
    """Records that first come back to pageable and later to page-locked
    memory, with the fault list shrinking and growing in between."""
    w = gen.generate(n_gates=600, n_pi=16, n_po=16, n_levels=15, n_patterns=100, seed=2, faults="pins")
    sim = Simulator(0)
    sim.read_text(w["ckt"], w["flst"], w["ptn"])
    site, pin, value = sim.faults()
    sim.run()
    want = sim.results().copy()
    order = np.random.default_rng(0).permutation(len(site))
    for n in (len(site), 50, len(site) // 2, len(site)):
        pick = order[:n]
        sim.set_faults(site[pick], pin[pick], value[pick])
        for k in range(150):
            sim.run()
            if k % 30 == 0 or k == 149:
                assert np.array_equal(sim.results(), want[pick])
