"""Affine alignments of targets of more bands than the boundary rows' epochs can
tell apart with two rows: homologies across the edges of the first bands and of
those after the epochs have come round, listed and unlisted pairs and the
unbatched form, maxima and hits against the oracle."""
import numpy as np
import pytest

import cases
from engine_helpers import configure, decode_hits
from pypaswas_b200 import _native, scores

pytestmark = pytest.mark.gpu


def _planted(rng, alphabet, lq, lt, places):
    """A query, and a target that holds mutated copies of it that start at `places`."""
    rs = lambda n: "".join(alphabet[i] for i in rng.integers(0, len(alphabet), n))
    q, t = rs(lq), rs(lt)
    for p in places:
        frag = cases.mutate(rng, q, alphabet, 0.04, 3)
        t = t[:p] + frag + t[p + len(frag):]
    return q, t[:lt]


def _check(engine_lib, oracle_mod, q, t, st, form):
    score = scores.make_score(st)
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        e.set_queries([s.encode() for s in q], np.arange(len(q)))
        e.set_targets([s.encode() for s in t], np.arange(len(t)) + len(q))
        if form == "listed":
            e.set_pairs(list(range(len(q))), list(range(len(t))))
        info = e.align(plain=form == "plain")
        pm = e.pair_max()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    assert info.score_path == (3 if form == "plain" else 2)
    found = 0
    for a in range(len(q)):
        for b in range(len(t)):
            if form == "listed" and a != b:
                continue
            ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), [q[a]], [t[b]],
                                 cases.pos_scores(score, st, [q[a]], [t[b]]), float(st.minimum_score))
            assert pm[a, b] == ref["pair_max"][0, 0]
            got = [h for h in hits if (h["query"], h["target"]) == (a, b)]
            assert got == [dict(h, query=a, target=b) for h in ref["hits"]]
            found += len(got)
    return found


@pytest.mark.parametrize("alphabet,settings", [
    ("ACGT", dict(match_score="5", mismatch_score="-8", gap_score="-12", gap_extension="-3", minimum_score="500",
                  lower_limit_score="0.9", filter_factor="0.1")),
    (cases.PROTEIN, dict(matrix_name="BLOSUM62", gap_score="-11", gap_extension="-1", minimum_score="500",
                         lower_limit_score="0.9", filter_factor="0.1"))])
@pytest.mark.parametrize("form", ["listed", "unlisted", "plain"])
def test_homologies_over_the_epochs_period(engine_lib, oracle_mod, alphabet, settings, form):
    rng = np.random.default_rng(len(alphabet))
    q, t = _planted(rng, alphabet, 750, 33700, [262, 32010, 32770])  # bands 1 to 3, 125 to 131
    assert _check(engine_lib, oracle_mod, [q], [t], cases.Settings(**settings), form) >= 3


@pytest.mark.parametrize("form", ["listed", "unlisted"])
def test_more_bands_than_warps(engine_lib, oracle_mod, form):
    # 641 bands: one block an SM has 592 warps, so that the last bands wait for earlier ones
    rng = np.random.default_rng(12)
    st = cases.Settings(match_score="5", mismatch_score="-8", gap_score="-12", gap_extension="-3",
                        minimum_score="250", lower_limit_score="0.7", filter_factor="0.1")
    q, t = zip(*[_planted(rng, "ACGT", 130, 164000, [200 + 64 * i, 700, 32200, 100300, 160900, 163300])
                 for i in range(2)])
    assert _check(engine_lib, oracle_mod, list(q), list(t), st, form) >= 12
