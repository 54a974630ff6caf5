"""A short pair of several bands beside a very long one, in one band sweep: the
short pair's maximum and hits against the oracle (its homology lies across the
band edge and below it)."""
import numpy as np
import pytest

import cases
from engine_helpers import configure, decode_hits
from pypaswas_b200 import _native, scores

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extension", ["0", "-1"])
@pytest.mark.parametrize("tile_trace", [0, 1])
def test_short_pair_beside_a_long_one(engine_lib, oracle_mod, extension, tile_trace):
    rng = np.random.default_rng(6)
    rs = lambda n: "".join(np.array(list("ACGT"))[rng.integers(0, 4, n)])
    short_q = rs(100)
    q = [rs(200000), short_q]
    t = [rs(400000), rs(225) + cases.mutate(rng, short_q, "ACGT", 0.03, 1) + rs(60) + short_q[20:80] + rs(30)]
    st = cases.Settings(gap_extension=extension, minimum_score="8", lower_limit_score="0.6")
    score = scores.make_score(st)
    ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), [q[1]], [t[1]],
                         cases.pos_scores(score, st, [q[1]], [t[1]]), float(st.minimum_score))
    assert len(ref["hits"]) >= 2
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        e.set_queries([s.encode() for s in q], np.arange(2))
        e.set_targets([s.encode() for s in t], np.arange(2) + 2)
        e.set_pairs([0, 1], [0, 1])
        e.set_tuning(_native.PW_TUNE_TILE_TRACE, tile_trace)
        info = e.align()
        pm = e.pair_max()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    assert info.score_path == 2
    assert pm[1, 1] == ref["pair_max"][0, 0]
    assert hits == [dict(h, query=1, target=1) for h in ref["hits"]]
