"""Scores-only calls of the 16-bit sweep end with their work done: the score
phase's time is reported and, with pairs past the 16-bit limit, holds the 32-bit
sweep of these pairs; the next call on the engine works."""
import numpy as np
import pytest

from engine_helpers import decode_hits
from pypaswas_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [64, 257, 258, 700])
def test_score_only_times_and_maxima(engine_lib, oracle_mod, length):
    rng = np.random.default_rng(length)
    bases = np.frombuffer(b"ACGT", np.uint8)
    q = [bytes(bases[rng.integers(0, 4, length)]) for _ in range(300)]
    t = [q[k] for k in range(40)]
    matrix = np.full((255, 255), -100.0, np.float32)
    np.fill_diagonal(matrix, 127.0)
    over = 127 * length >= 32640
    p = oracle_mod.OracleParams(matrix, 1, -100.0, 0.0, False, 1.0, 1.0e6)
    want = oracle_mod.pair_max(p, [s.decode() for s in q[:45]], [s.decode() for s in t])
    e = _native.Engine(0, lib=engine_lib)
    try:
        e.set_scoring(matrix, 1, -100.0, 0.0, False, 1.0, 127.0 * length, 127.0 * length, 127.0, 0.05)
        e.set_queries(q, np.arange(len(q)))
        e.set_targets(t, np.arange(len(t)) + len(q))
        for _ in range(8):
            info = e.align(score_only=True)
            assert info.score_path == 0 and info.overflow_pairs == (40 if over else 0)
            # the phase's interval holds its kernels' (the events are read in microseconds)
            assert info.score_ms >= info.score_kernel_ms * 0.999 > 0
            assert info.total_ms >= info.score_ms * 0.9
            np.testing.assert_array_equal(e.pair_max()[:45], want)
        info = e.align()
        assert info.hits == len(decode_hits(*e.hits())) == 40
    finally:
        e.close()
