"""The 16-bit halves of the checkpointing band sweep: gaps at and past the 16-bit
range (listed pairs that share a query and a target length, and the same pairs
as an unlisted call of few long sequences), against the oracle; maxima around the
16-bit limit when the caller's highest score is not the matrix's."""
import numpy as np
import pytest

from engine_helpers import decode_hits
from pypaswas_b200 import _native

pytestmark = pytest.mark.gpu


def _matrix(match, mismatch):
    m = np.full((255, 255), mismatch, np.float32)
    np.fill_diagonal(m, match)
    return m


def _engine(lib, q, t, matrix, gap, minimum, highest, pairs):
    e = _native.Engine(0, lib=lib)
    e.set_scoring(matrix, 1, gap, 0.0, False, 1.0, minimum, minimum, highest, 0.02)
    e.set_queries(q, np.arange(len(q)))
    e.set_targets(t, np.arange(len(t)) + len(q))
    if pairs:
        e.set_pairs([a for a, _ in pairs], [b for _, b in pairs])
    return e


def _bases(rng, n):
    return bytes(np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, n)])


@pytest.mark.parametrize("gap", [-5, -32767, -32768, -32769, -40000, -65536, -100000, -1000000])
@pytest.mark.parametrize("listed", [True, False])
def test_gaps_past_16_bits(engine_lib, oracle_mod, gap, listed):
    rng = np.random.default_rng(3)
    n = 600 if listed else 4200  # unlisted: from 2^24 cells on band by band
    q = [_bases(rng, n)]
    core = q[0][n // 3:n // 3 + 200]
    t = [_bases(rng, 300) + core + _bases(rng, n - 500),
         _bases(rng, 200) + core[:100] + _bases(rng, 3) + core[100:] + _bases(rng, n - 403)]
    pairs = [(0, 0), (0, 1)]
    matrix = _matrix(5.0, -3.0)
    p = oracle_mod.OracleParams(matrix, 1, float(gap), 0.0, False, 1.0, 60.0)
    e = _engine(engine_lib, q, t, matrix, float(gap), 60.0, 5.0, pairs if listed else None)
    try:
        info = e.align()
        pm = e.pair_max()
        hits = decode_hits(*e.hits())
    finally:
        e.close()
    assert info.score_path == 2 and (info.paired_cells > 0) == (gap >= -32768)
    for a, b in pairs:
        pos = np.array([[np.float32(5.0 * min(len(q[a]), len(t[b])) * 0.02)]], np.float32)
        ref = oracle_mod.run(p, [q[a].decode()], [t[b].decode()], pos, 60.0)
        assert pm[a, b] == ref["pair_max"][0, 0]
        assert [h for h in hits if h["target"] == b] == [dict(h, query=a, target=b) for h in ref["hits"]]


@pytest.mark.parametrize("highest", [-3.0, 1.0, 127.0, 1.0e6, 1.0e12])
@pytest.mark.parametrize("length", [256, 257, 258, 259, 400])
def test_limit_is_the_matrix_own(engine_lib, highest, length):
    # identical sequences: the maximum is 127 a residue; 258 of them are past the limit
    q = [_bases(np.random.default_rng(length), length)]
    e = _engine(engine_lib, q, [q[0], q[0]], _matrix(127.0, -100.0), -100.0, 1.0e9, highest, [(0, 0), (0, 1)])
    try:
        info = e.align(score_only=True)
        pm = e.pair_max()
    finally:
        e.close()
    assert info.overflow_pairs == (2 if length >= 258 else 0)
    assert pm.tolist() == [[127.0 * length] * 2]
