"""The tuned sweep shape and the pattern count: a shape timed on few patterns
is reconsidered for more."""
import numpy as np
import pytest

from lsim_b200 import Simulator, gen
from tests.oracle_lib import Oracle

pytestmark = pytest.mark.gpu


def test_a_shape_tuned_on_few_patterns_is_reconsidered():
    w = gen.generate(n_gates=2000, n_pi=64, n_po=64, n_levels=30, n_patterns=4096, seed=5)
    sim = Simulator(0)
    sim.read_text(w["ckt"], w["flst"], w["ptn"])
    words = sim.patterns()
    ref = Oracle(w["ckt"], w["flst"], w["ptn"]).simulate()
    tuned = []
    for P in (64, 64, 512, 192, 448, 1024, 1088, 2048, 4096, 64):
        sim.set_patterns(words[:P // 64], P)
        sim.run(tune=True)
        tuned.append(sim.stats()["ms_tune"] > 0)
        if P == 4096:
            got = sim.results()
            assert np.array_equal(got["count"], ref["count"])
            assert np.array_equal(got["first_pattern"], ref["first"])
    # 1, 1, 8, 3, 7, 16, 17, 32, 32 and 1 words a tile
    assert tuned == [True, False, True, False, False, True, True, False, False, False]
