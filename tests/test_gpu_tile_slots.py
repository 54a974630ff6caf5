"""Tiles of codes computed ahead of the walks: every tile of the path listed,
some of them (few slots, so that the walk computes the rest), and paths that
leave the listed corridor (long insertions), against the oracle."""
import numpy as np
import pytest

import cases
from engine_helpers import configure, decode_hits
from pypaswas_b200 import _native, scores

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wave_limit", [0, 1 << 16, 1 << 20])
@pytest.mark.parametrize("pairs_given", [True, False])
@pytest.mark.parametrize("shift", [0, 90])
def test_walks_with_all_some_and_no_tiles_ahead(engine_lib, oracle_mod, wave_limit, pairs_given, shift):
    rng = np.random.default_rng(shift + 1)
    rs = lambda n: "".join("ACGT"[i] for i in rng.integers(0, 4, n))
    st = cases.Settings(match_score="5", mismatch_score="-3", gap_score="-1", minimum_score="60",
                        filter_factor="0.02", lower_limit_score="0.97")
    score = scores.make_score(st)
    q, t = [], []
    for n in (700, 1500, 2100):
        a = rs(n)
        b = cases.mutate(rng, a, "ACGT", 0.05, n // 60)
        for p in (n // 4, n // 2, 3 * n // 4):  # gaps that move the path off its diagonal
            b = b[:p] + rs(shift) + b[p:]
        q.append(a)
        t.append(b)
    ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), q, t, cases.pos_scores(score, st, q, t),
                         float(st.minimum_score))
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        e.set_queries([s.encode() for s in q], np.arange(len(q)))
        e.set_targets([s.encode() for s in t], np.arange(len(t)) + len(q))
        e.set_wave_limit(wave_limit)
        if pairs_given:
            e.set_pairs(np.repeat(np.arange(3), 3), np.tile(np.arange(3), 3))
        info = e.align(int32=not pairs_given)  # (the 32-bit sweep: a few long sequences go band by band otherwise)
        pm = e.pair_max()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    assert info.tile_pairs > 0 and info.score_path == (2 if pairs_given else 1)
    np.testing.assert_array_equal(pm, ref["pair_max"])
    assert hits == ref["hits"]
