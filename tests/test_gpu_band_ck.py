"""The checkpointing band sweep of listed pairs (blocks of 4 columns, groups of
32, tiles of 128, bands of 256 rows) at lengths around each of these edges, two
pairs a warp and alone, against the oracle pair by pair: maxima and hits, which
come from the tiles recomputed from its checkpoints."""
import numpy as np
import pytest

import cases
from engine_helpers import configure, decode_hits
from pypaswas_b200 import _native, scores

pytestmark = pytest.mark.gpu
EDGES = [1, 3, 4, 5, 31, 32, 33, 127, 128, 129, 132, 255, 256, 257, 260, 385, 511, 512, 513, 700]


@pytest.mark.parametrize("alphabet,settings", [
    ("ACGT", dict(minimum_score="6", filter_factor="0.05")),
    (cases.PROTEIN, dict(matrix_name="BLOSUM62", gap_score="-8", minimum_score="25", filter_factor="0.01"))])
@pytest.mark.parametrize("paired", [True, False])
def test_edge_lengths(engine_lib, oracle_mod, alphabet, settings, paired):
    rng = np.random.default_rng(len(alphabet) + paired)
    st = cases.Settings(**settings)
    score = scores.make_score(st)

    def rs(n):
        return "".join(alphabet[i] for i in rng.integers(0, len(alphabet), n))

    q, t, pairs = [], [], []
    for i, n in enumerate(EDGES):
        m = EDGES[(7 * i + 3) % len(EDGES)]
        q.append(rs(n))
        for copy in range(2 if paired else 1):  # two targets of one length share a sweep
            k = min(n, m) // 2
            frag = cases.mutate(rng, q[-1][n - k:], alphabet, 0.1, k // 40)[:m]
            p = int(rng.integers(0, m - len(frag) + 1))
            s = rs(m)
            t.append(s[:p] + frag + s[p + len(frag):])
            pairs.append((i, len(t) - 1))
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        e.set_queries([s.encode() for s in q], np.arange(len(q)))
        e.set_targets([s.encode() for s in t], np.arange(len(t)) + len(q))
        e.set_pairs([a for a, _ in pairs], [b for _, b in pairs])
        info = e.align()
        pm = e.pair_max()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    assert info.score_path == 2 and (info.paired_cells > 0) == paired
    got = {}
    for h in hits:
        got.setdefault((h["query"], h["target"]), []).append(h)
    for a, b in pairs:
        ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), [q[a]], [t[b]],
                             cases.pos_scores(score, st, [q[a]], [t[b]]), float(st.minimum_score))
        assert pm[a, b] == ref["pair_max"][0, 0]
        assert got.get((a, b), []) == [dict(h, query=a, target=b) for h in ref["hits"]]


MANY_EDGES = [1, 4, 5, 7, 8, 9, 63, 64, 65, 121, 127, 128, 129, 135, 136, 248, 249, 256, 260, 384, 389, 513]


@pytest.mark.parametrize("paired", [True, False])
def test_many_bands(engine_lib, oracle_mod, paired):
    """More bands than warps in flight (two blocks an SM, warps that take band
    after band), beside pairs around the edges of blocks, groups and tiles."""
    st = cases.Settings(minimum_score="6", filter_factor="0.05")
    score = scores.make_score(st)
    rng = np.random.default_rng(41 + paired)

    def rs(n):
        return "".join("ACGT"[i] for i in rng.integers(0, 4, n))

    q, t, pairs = [], [], []
    for i, n in enumerate(MANY_EDGES):
        m = MANY_EDGES[(5 * i + 2) % len(MANY_EDGES)] + 256 * (i % 3)
        q.append(rs(n))
        for copy in range(2 if paired else 1):
            k = min(n, m) // 2
            frag = cases.mutate(rng, q[-1][n - k:], "ACGT", 0.1, k // 40)[:m]
            p = int(rng.integers(0, m - len(frag) + 1))
            s = rs(m)
            t.append(s[:p] + frag + s[p + len(frag):])
            pairs.append((i, len(t) - 1))
    checked = len(pairs)
    first, filler = len(t), 2 if paired else 1
    t += [rs(1024) for _ in range(filler)]  # four bands a chain
    for _ in range(700):
        q.append(rs(13))
        pairs += [(len(q) - 1, first + copy) for copy in range(filler)]
    checked_filler = list(range(checked, len(pairs), 97))
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        e.set_queries([s.encode() for s in q], np.arange(len(q)))
        e.set_targets([s.encode() for s in t], np.arange(len(t)) + len(q))
        e.set_pairs([a for a, _ in pairs], [b for _, b in pairs])
        info = e.align()
        pm = e.pair_max()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    assert info.score_path == 2 and (info.paired_cells > 0) == paired
    got = {}
    for h in hits:
        got.setdefault((h["query"], h["target"]), []).append(h)
    for k in [*range(checked), *checked_filler]:
        a, b = pairs[k]
        ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), [q[a]], [t[b]],
                             cases.pos_scores(score, st, [q[a]], [t[b]]), float(st.minimum_score))
        assert pm[a, b] == ref["pair_max"][0, 0]
        assert got.get((a, b), []) == [dict(h, query=a, target=b) for h in ref["hits"]]
