"""Calls that fail while a set's copies and encodings are under way, followed at
once by a call with other sets in the same page-locked arrays: its results are
the oracle's, and the failed call's message is the first invalid residue's."""
import numpy as np
import pytest

from pypaswas_b200 import _native
from pypaswas_b200.exceptions import InvalidOptionException

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_targets,length", [(40, 60), (3000, 80), (20000, 150)])
def test_sets_after_a_failed_call(engine_lib, oracle_mod, n_targets, length):
    rng = np.random.default_rng(n_targets)
    bases = np.frombuffer(b"ACGT", np.uint8)
    draw = lambda n, lo: [bytes(bases[rng.integers(0, 4, int(k))]) for k in rng.integers(lo, length, n)]
    matrix = np.full((200, 200), -3.0, np.float32)  # residue codes 1 .. 200
    np.fill_diagonal(matrix, 2.0)
    p = oracle_mod.OracleParams(matrix, 1, -4.0, 0.0, False, 1.0, 1.0e6)
    e = _native.Engine(0, lib=engine_lib)
    try:
        e.set_scoring(matrix, 1, -4.0, 0.0, False, 1.0, 1.0e6, 1.0e6, 2.0, 0.05)
        for turn in range(6):
            e.set_targets(draw(n_targets, 20), np.arange(n_targets) + 3)
            e.set_queries([b"ACGT", b"AC\xf0T"], np.arange(2))
            with pytest.raises(InvalidOptionException, match="code 240"):
                e.align(score_only=True)
            targets, queries = draw(n_targets, 10), draw(3, 20)
            e.set_targets(targets, np.arange(n_targets) + 3)
            e.set_queries(queries, np.arange(3))
            e.align(score_only=True)
            want = oracle_mod.pair_max(p, [s.decode() for s in queries], [s.decode() for s in targets[:400]])
            np.testing.assert_array_equal(e.pair_max()[:, :400], want)
    finally:
        e.close()
