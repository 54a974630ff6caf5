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
