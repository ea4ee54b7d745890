"""Handles, batches and their kernels' limits in several threads at once."""
import threading

import numpy as np
import pytest

from lsim_b200 import Simulator, gen
from lsim_b200.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [False, True])
def test_threads_with_circuits_of_different_slots(batch):
    """Each thread its own circuit at 8 words an item, 10 to 80 KB of slots."""
    failed = []

    def work(gates, levels):
        try:
            w = gen.generate(n_gates=gates, n_pi=64, n_po=64, n_levels=levels, n_patterns=64, seed=1)
            sim = Simulator(-1 if batch else 0)
            sim.read_text(w["ckt"], w["flst"], w["ptn"])
            runner = Batch(0) if batch else sim
            if batch:
                runner.add(sim)
            want = None
            for k in range(300):
                # graphs off, so that every run sets the limits and launches
                runner.run(words_per_item=8, **(dict(graph=False, block_threads=64 + 64 * (k % 2)) if batch else {}))
                got = sim.results()
                want = got.copy() if want is None else want
                assert np.array_equal(got, want)
        except Exception as e:  # noqa: BLE001
            failed.append("%d gates: %s" % (gates, e))

    threads = [threading.Thread(target=work, args=a)
               for a in ((600, 20), (4000, 12), (700, 24), (5000, 15), (800, 28), (4500, 11), (900, 16), (6000, 18))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
