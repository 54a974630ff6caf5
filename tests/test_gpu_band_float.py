"""Traced pairs with fractional scores: the fp32 band direction sweep at lengths
around its lanes (8 rows), bands (256 rows) and blocks (32 columns), linear and
affine gap, against the oracle; large alphabets, whose profiles leave room for
fewer warps a block, on every band sweep."""
import numpy as np
import pytest

import cases
from engine_helpers import configure, decode_hits
from pypaswas_b200 import _native, scores

pytestmark = pytest.mark.gpu
EDGES = [1, 7, 8, 9, 31, 32, 33, 64, 65, 150, 255, 256, 257, 300, 513]


@pytest.mark.parametrize("affine", [False, True])
@pytest.mark.parametrize("matrix", ["DNA-RNA", "BLOSUM62"])
def test_edge_lengths(engine_lib, oracle_mod, affine, matrix):
    rng = np.random.default_rng(7 + affine)
    st = cases.Settings(matrix_name=matrix, match_score="1.5", mismatch_score="-2.25", gap_score="-3.5",
                        gap_extension="-0.75" if affine else "0", minimum_score="5", lower_limit_score="0.9",
                        filter_factor="0.02")
    alphabet = "ACGT" if matrix == "DNA-RNA" else cases.PROTEIN
    score = scores.make_score(st)
    rs = lambda n: "".join(alphabet[i] for i in rng.integers(0, len(alphabet), n))
    q = [rs(n) for n in EDGES]
    t = []
    for i, n in enumerate(EDGES):
        m = EDGES[(4 * i + 3) % len(EDGES)]
        k = min(n, m) // 2
        frag = cases.mutate(rng, q[i][n - k:], alphabet, 0.1, k // 40)[:m]
        p = int(rng.integers(0, m - len(frag) + 1))
        s = rs(m)
        t.append(s[:p] + frag + s[p + len(frag):])
    ref = oracle_mod.run(cases.oracle_params(oracle_mod, score), q, t, cases.pos_scores(score, st, q, t),
                         float(st.minimum_score))
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        e.set_queries([s.encode() for s in q], np.arange(len(q)))
        e.set_targets([s.encode() for s in t], np.arange(len(t)) + len(q))
        info = e.align()
        pm = e.pair_max()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    assert info.warp_pairs == info.traced_pairs > 0 and info.score_path == 1
    np.testing.assert_array_equal(pm, ref["pair_max"])
    assert hits == ref["hits"]


@pytest.mark.parametrize("residues", [60, 120, 225])
@pytest.mark.parametrize("gap,ext", [(-4.0, 0.0), (-4.0, -1.0), (-2.5, 0.0), (-2.5, -0.5)])
def test_large_alphabets(engine_lib, oracle_mod, residues, gap, ext):
    rng = np.random.default_rng(residues)
    letters = np.concatenate([np.arange(1, 97), np.arange(123, 256)])[:residues]  # no lower-case letters
    matrix = np.full((255, 255), -3.0, np.float32)
    np.fill_diagonal(matrix, 4.0)
    q = [bytes(rng.choice(letters, n).astype(np.uint8)) for n in (700, 300, 64)]
    t = [q[0][100:500] + q[1][:40], q[1][50:] + q[0][:200], q[2], q[2][::-1]]
    pairs = [(0, 0), (1, 1), (2, 2), (2, 3)]
    e = _native.Engine(0, lib=engine_lib)
    try:
        e.set_scoring(matrix, 1, gap, ext, ext != 0, 1.0, 20.0, 20.0, 4.0, 0.05)
        e.set_queries(q, np.arange(3))
        e.set_targets(t, np.arange(4) + 3)
        p = oracle_mod.OracleParams(matrix, 1, gap, ext, ext != 0, 1.0, 20.0)
        want = oracle_mod.pair_max(p, [s.decode("latin-1") for s in q], [s.decode("latin-1") for s in t])
        for listed in (True, False):
            if listed:
                e.set_pairs([a for a, _ in pairs], [b for _, b in pairs])
            else:
                e.set_pairs([], [])
            info = e.align()
            pm = e.pair_max()
            assert info.traced_pairs > 0 and info.hits > 0
            for a, b in pairs:
                assert pm[a, b] == want[a, b]
    finally:
        e.close()
