"""Hit order and strings: alignments around the lengths where a thread, a warp or
a block spells them, few and many hits, keys within and beyond 64 bits, against
the oracle."""
import numpy as np
import pytest

import cases
from engine_helpers import run_engine
from pypaswas_b200 import scores

pytestmark = pytest.mark.gpu


def _check(engine_lib, oracle_mod, q, t, st, least):
    score = scores.make_score(st)
    ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), q, t, cases.pos_scores(score, st, q, t),
                         float(st.minimum_score))
    pm, hits, info, _ = run_engine(engine_lib, q, t, score, st)
    np.testing.assert_array_equal(pm, ref["pair_max"])
    assert len(hits) >= least and hits == ref["hits"]


@pytest.mark.parametrize("lengths", [[31, 32, 33, 64, 65], [511, 513, 2047, 2048, 2049, 2600]])
def test_alignment_lengths(engine_lib, oracle_mod, lengths):
    rng = np.random.default_rng(len(lengths))
    base = ["".join("ACGT"[i] for i in rng.integers(0, 4, n)) for n in lengths]
    t = [s[:len(s) // 2] + "G" + s[len(s) // 2:] for s in base] + base
    _check(engine_lib, oracle_mod, base, t, cases.Settings(match_score="3", gap_score="-4", minimum_score="40"),
           2 * len(lengths))


@pytest.mark.parametrize("n", [30, 34])  # 900 and 1,156 hits: either side of one block
@pytest.mark.parametrize("match", ["1", "1.5"])
def test_few_and_many_hits(engine_lib, oracle_mod, n, match):
    rng = np.random.default_rng(n)
    s = "".join("ACGT"[i] for i in rng.integers(0, 4, 35))
    vary = lambda k: s[:k % 30] + "ACGT"[k % 4] + s[k % 30 + 1:]
    _check(engine_lib, oracle_mod, [vary(k) for k in range(n)], [vary(3 * k + 1) for k in range(n)],
           cases.Settings(match_score=match, minimum_score="10"), n * n)


def test_keys_beyond_64_bits(engine_lib, oracle_mod):
    # fp32 scores (32 bits) and positions up to 70,000 (14 + 14 bits)
    rng = np.random.default_rng(3)
    rs = lambda n: "".join("ACGT"[i] for i in rng.integers(0, 4, n))
    t = [rs(40) for _ in range(20)]
    q = [rs(69000) + "".join(t[:10])] + [s[3:] for s in t]
    _check(engine_lib, oracle_mod, q, t, cases.Settings(match_score="1.5", minimum_score="30"), 20)
