"""Pattern blocks whose last tile is not full: the sweeps take only the
words that hold patterns.  Sizes at the edges of a word, of the words of one
sweep item and of a tile, bit-exact against the oracle."""
import numpy as np
import pytest

from lsim_b200 import Simulator, gen
from lsim_b200.batch import Batch
from tests.oracle_lib import Oracle

pytestmark = pytest.mark.gpu

SIZES = [1, 64, 65, 128, 129, 8 * 64, 8 * 64 + 1, 31 * 64, 2048, 2049, 2048 + 5 * 64 + 3, 4096]


def _work(P):
    return gen.generate(n_gates=350, n_pi=14, n_po=9, n_levels=11, n_patterns=P, seed=P % 7,
                        type_mask=gen.ALL_TYPES if P % 2 else gen.BENCH_TYPES, faults="pins")


def _same(got, ref):
    assert np.array_equal(got["detected"], ref["detected"])
    assert np.array_equal(got["first_pattern"], ref["first"])
    assert np.array_equal(got["count"], ref["count"])
    assert np.array_equal(got["ref_last_round_flag"], ref["ref_flag"])


@pytest.mark.parametrize("P", SIZES)
def test_plain_sweeps(P):
    w = _work(P)
    ref = Oracle(w["ckt"], w["flst"], w["ptn"]).simulate()
    sim = Simulator(0)
    sim.read_text(w["ckt"], w["flst"], w["ptn"])
    for opts in [dict()] + [dict(words_per_item=m) for m in (1, 2, 4, 8)] + \
            [dict(sweep_variant="global", words_per_item=m) for m in (1, 2)]:
        sim.run(**opts)
        _same(sim.results(), ref)


def test_batch_of_all_sizes():
    sims, refs = [], []
    with Batch(0) as b:
        for P in SIZES:
            w = _work(P)
            s = Simulator(-1)
            s.read_text(w["ckt"], w["flst"], w["ptn"])
            sims.append(s)
            refs.append(Oracle(w["ckt"], w["flst"], w["ptn"]).simulate())
            b.add(s)
        for m in (0, 1, 2, 4, 8):
            b.run(words_per_item=m)
            for s, ref in zip(sims, refs):
                _same(s.results(), ref)


@pytest.mark.parametrize("n_words", [1, 2, 147, 148, 149, 296, 297, 592, 593, 1200])
@pytest.mark.parametrize("gates,levels", [(300, 12), (9000, 3)])
def test_good_machine_word_counts(n_words, gates, levels):
    """Good-machine values at the edges of the words per CTA, narrow levels
    (all levels in one launch) and wide ones, against the oracle."""
    P = 64 * n_words - 5
    w = gen.generate(n_gates=gates, n_pi=20, n_po=15, n_levels=levels, n_patterns=P, seed=n_words,
                     type_mask=gen.ALL_TYPES)
    sim = Simulator(0)
    sim.read_text(w["ckt"], "0\n", w["ptn"])
    sim.run()
    ref = Oracle(w["ckt"], "0\n", w["ptn"])
    for rd in sorted({0, n_words // 2, n_words - 1}):
        assert np.array_equal(sim.good_values(rd), ref.good_values(rd)), rd
