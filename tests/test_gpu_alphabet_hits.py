"""Hits of large alphabets, whose profiles leave room for fewer warps a block on
the band sweeps (linear and affine, whole and fractional scores), listed and
unlisted, against the oracle pair by pair."""
import numpy as np
import pytest

from engine_helpers import decode_hits
from pypaswas_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("residues", [60, 120, 225])
@pytest.mark.parametrize("gap,ext", [(-4.0, 0.0), (-4.0, -1.0), (-2.5, 0.0), (-2.5, -0.5)])
@pytest.mark.parametrize("listed", [True, False])
def test_hits(engine_lib, oracle_mod, residues, gap, ext, listed):
    rng = np.random.default_rng(residues + listed)
    letters = np.concatenate([np.arange(1, 97), np.arange(123, 256)])[:residues]  # no lower-case letters
    matrix = np.full((255, 255), -3.0, np.float32)
    np.fill_diagonal(matrix, 4.0)
    draw = lambda n: bytes(rng.choice(letters, n).astype(np.uint8))
    q = [draw(n) for n in (700, 300, 64)]
    cut = lambda s, a, b: s[a:(a + b) // 2] + draw(2) + s[(a + b) // 2 + 1:b]  # a gap and a mismatch
    t = [draw(150) + cut(q[0], 100, 500) + q[1][:40], cut(q[1], 50, 300) + q[0][:200], q[2], q[2][::-1] + draw(260)]
    pairs = [(0, 0), (1, 1), (2, 2), (2, 3)]
    p = oracle_mod.OracleParams(matrix, 1, gap, ext, ext != 0, 0.9, 20.0)
    e = _native.Engine(0, lib=engine_lib)
    try:
        e.set_scoring(matrix, 1, gap, ext, ext != 0, 0.9, 20.0, 20.0, 4.0, 0.05)
        e.set_queries(q, np.arange(3))
        e.set_targets(t, np.arange(4) + 3)
        if listed:
            e.set_pairs([a for a, _ in pairs], [b for _, b in pairs])
        info = e.align()
        pm = e.pair_max()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    assert info.traced_pairs > 0
    found = 0
    for a, b in pairs if listed else [(a, b) for a in range(3) for b in range(4)]:
        pos = np.array([[np.float32(4.0 * min(len(q[a]), len(t[b])) * 0.05)]], np.float32)
        ref = oracle_mod.run(p, [q[a].decode("latin-1")], [t[b].decode("latin-1")], pos, 20.0)
        assert pm[a, b] == ref["pair_max"][0, 0]
        assert [h for h in hits if (h["query"], h["target"]) == (a, b)] == \
            [dict(h, query=a, target=b) for h in ref["hits"]]
        found += len(ref["hits"])
    assert found >= 3
