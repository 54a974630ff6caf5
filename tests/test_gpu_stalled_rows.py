"""The band sweeps that hand rows down in self-validating words give up, within
the wait limit, on a row that nobody stores (PW_TUNE_STALL_TEST 2): the polls of
the checkpointing sweep (two pairs a warp and alone) and of the affine sweep
(maxima and cell codes).  The next call on the same engine is the oracle's."""
import time

import numpy as np
import pytest

import cases
from engine_helpers import configure, decode_hits
from pypaswas_b200 import _native, scores
from pypaswas_b200.exceptions import CudaException

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sweep", ["paired", "single", "affine maxima", "affine codes"])
def test_poll_runs_out_and_engine_recovers(engine_lib, oracle_mod, sweep):
    rng = np.random.default_rng(3)
    rs = lambda n: "".join("ACGT"[i] for i in rng.integers(0, 4, n))
    listed = sweep != "affine codes"
    n = 3 if listed else 320  # enough for the all-against-all score sweep
    q = [rs(90 + k % 40) for k in range(n)]
    # two targets of one length, five bands each
    t = [rs(700) + cases.mutate(rng, q[k], "ACGT", 0.05, 1) + rs(400) for k in range(2)]
    t[1] = (t[1] + rs(1300))[:len(t[0])] + ("" if sweep == "paired" else "A")
    st = cases.Settings(minimum_score="25", gap_extension="-1" if sweep.startswith("affine") else "0")
    score = scores.make_score(st)
    pairs = [(0, 0), (0, 1), (1, 0), (1, 1), (2, 0)]
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        e.set_queries([s.encode() for s in q], np.arange(n))
        e.set_targets([s.encode() for s in t], np.arange(2) + n)
        if listed:
            e.set_pairs([a for a, _ in pairs], [b for _, b in pairs])
        first = e.align()
        want_pm, want = e.pair_max(), decode_hits(*e.hits())
        assert first.score_path == (2 if listed else 0) and first.warp_pairs + first.tile_pairs > 0
        assert (first.paired_cells > 0) == (sweep == "paired")
        e.set_tuning(_native.PW_TUNE_WAIT_NS, 5_000_000)
        e.set_tuning(_native.PW_TUNE_STALL_TEST, 2)
        began = time.monotonic()
        with pytest.raises(CudaException, match="a band waited too long"):
            e.align()
        assert time.monotonic() - began < 2.0
        e.set_tuning(_native.PW_TUNE_WAIT_NS, 0)
        e.align()
        np.testing.assert_array_equal(e.pair_max(), want_pm)
        assert decode_hits(*e.hits()) == want
    finally:
        e.close()
    for a, b in pairs:
        ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), [q[a]], [t[b]],
                             cases.pos_scores(score, st, [q[a]], [t[b]]), float(st.minimum_score))
        assert want_pm[a, b] == ref["pair_max"][0, 0]
        assert [h for h in want if (h["query"], h["target"]) == (a, b)] == \
            [dict(h, query=a, target=b) for h in ref["hits"]]
