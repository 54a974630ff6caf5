"""The affine band sweep (blocks of 2 columns, groups of 32, bands of 256 rows)
at lengths around these edges and over many bands (the row words' epochs
repeat after 126 bands), as listed pairs (maxima, then codes) and traced from
an all-against-all call, against the oracle: maxima and hits."""
import numpy as np
import pytest

import cases
from engine_helpers import configure, decode_hits
from pypaswas_b200 import _native, scores

pytestmark = pytest.mark.gpu
EDGES = [1, 2, 3, 31, 32, 33, 34, 63, 65, 255, 256, 257, 258, 511, 512, 513, 700, 769]


def _check(engine_lib, oracle_mod, q, t, pairs, st, **align):
    score = scores.make_score(st)
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        e.set_queries([s.encode() for s in q], np.arange(len(q)))
        e.set_targets([s.encode() for s in t], np.arange(len(t)) + len(q))
        if pairs:
            e.set_pairs([a for a, _ in pairs], [b for _, b in pairs])
        info = e.align(**align)
        pm = e.pair_max()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    got = {}
    for h in hits:
        got.setdefault((h["query"], h["target"]), []).append(h)
    for a, b in pairs or [(a, b) for a in range(len(q)) for b in range(len(t))]:
        ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), [q[a]], [t[b]],
                             cases.pos_scores(score, st, [q[a]], [t[b]]), float(st.minimum_score))
        assert pm[a, b] == ref["pair_max"][0, 0]
        assert got.get((a, b), []) == [dict(h, query=a, target=b) for h in ref["hits"]]
    return info


def _case(rng, alphabet, lens_q, lens_t):
    rs = lambda n: "".join(alphabet[i] for i in rng.integers(0, len(alphabet), n))
    q, t = [], []
    for n, m in zip(lens_q, lens_t):
        q.append(rs(n))
        k = min(n, m) // 2
        frag = cases.mutate(rng, q[-1][n - k:], alphabet, 0.1, k // 40)[:m]
        p = int(rng.integers(0, m - len(frag) + 1))
        s = rs(m)
        t.append(s[:p] + frag + s[p + len(frag):])
    return q, t


@pytest.mark.parametrize("alphabet,settings", [
    ("ACGT", dict(gap_score="-2", gap_extension="-1", minimum_score="6", filter_factor="0.05")),
    (cases.PROTEIN, dict(matrix_name="BLOSUM62", gap_score="-11", gap_extension="-1", minimum_score="25",
                         filter_factor="0.01", lower_limit_score="0.95"))])
@pytest.mark.parametrize("listed", [True, False])
def test_edge_lengths(engine_lib, oracle_mod, alphabet, settings, listed):
    rng = np.random.default_rng(len(alphabet) + listed)
    n = len(EDGES)
    q, t = _case(rng, alphabet, EDGES, [EDGES[(7 * i + 5) % n] for i in range(n)])
    info = _check(engine_lib, oracle_mod, q, t, [(i, i) for i in range(n)] if listed else None,
                  cases.Settings(**settings))
    assert info.warp_pairs > 0 and info.score_path == 2  # (few long sequences go band by band unlisted too)


def test_many_bands(engine_lib, oracle_mod):
    # 141 bands: ring slots reused 70 times, past the epochs' period of 63
    rng = np.random.default_rng(5)
    q, t = _case(rng, "ACGT", [150, 90], [36000, 33000])
    st = cases.Settings(gap_score="-3", gap_extension="-1", minimum_score="20", filter_factor="0.1")
    info = _check(engine_lib, oracle_mod, q, t, [(0, 0), (1, 1)], st)
    assert info.score_path == 2


@pytest.mark.parametrize("affine", [True, False])
@pytest.mark.parametrize("limit", ["0.5", "0.9"])
def test_walks_with_many_candidates(engine_lib, oracle_mod, affine, limit):
    # repeats: candidates that cover one another, walks that meet, stop cells
    # with and without a candidate on their run (a warp a pair; linear: stored codes)
    rng = np.random.default_rng(9)
    rs = lambda n: "".join("ACGT"[i] for i in rng.integers(0, 4, n))
    unit = rs(45)
    q, t = [], []
    for n in (120, 330, 600):
        q.append(rs(n) + unit + rs(20) + unit[:30] + rs(n // 3))
        t.append(rs(n // 2) + cases.mutate(rng, unit, "ACGT", 0.08, 1) + rs(31) + unit + rs(n))
    st = cases.Settings(match_score="5", mismatch_score="-3", gap_score="-4", gap_extension="-1" if affine else "0",
                        minimum_score="40", lower_limit_score=limit, filter_factor="0.02")
    score = scores.make_score(st)
    ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), q, t, cases.pos_scores(score, st, q, t),
                         float(st.minimum_score))
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        e.set_queries([s.encode() for s in q], np.arange(len(q)))
        e.set_targets([s.encode() for s in t], np.arange(len(t)) + len(q))
        e.set_tuning(_native.PW_TUNE_TILE_TRACE, 1)
        info = e.align()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    assert info.warp_pairs > 0 and info.starting_points > info.traced_pairs
    assert hits == ref["hits"]


def test_many_chains(engine_lib, oracle_mod):
    """More bands than warps in flight with one block an SM (two and more blocks,
    warps that take band after band): maxima and hits of a sample."""
    st = cases.Settings(matrix_name="BLOSUM62", gap_score="-11", gap_extension="-1", minimum_score="25",
                        filter_factor="0.01")
    score = scores.make_score(st)
    rng = np.random.default_rng(77)

    def rs(n):
        return "".join(cases.PROTEIN[i] for i in rng.integers(0, len(cases.PROTEIN), n))

    n = 900
    q = [rs(int(rng.integers(20, 60))) for _ in range(n)]
    t = [rs(int(rng.integers(600, 1000))) for _ in range(8)]  # three or four bands
    t = [s[:250] + q[k][:20] + s[270:510] + q[k + 8][:20] + s[530:] for k, s in enumerate(t)]
    pairs = [(i, i % 8) for i in range(n)]
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        e.set_queries([s.encode() for s in q], np.arange(n))
        e.set_targets([s.encode() for s in t], np.arange(8) + n)
        e.set_pairs([a for a, _ in pairs], [b for _, b in pairs])
        info = e.align()
        pm = e.pair_max()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    assert info.score_path == 2
    for k in [*range(16), *range(16, n, 59)]:
        a, b = pairs[k]
        ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), [q[a]], [t[b]],
                             cases.pos_scores(score, st, [q[a]], [t[b]]), float(st.minimum_score))
        assert pm[a, b] == ref["pair_max"][0, 0]
        assert [h for h in hits if (h["query"], h["target"]) == (a, b)] == \
            [dict(h, query=a, target=b) for h in ref["hits"]]
