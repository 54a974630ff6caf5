"""The 16-bit score sweep's forms (profile layout by alphabet size, strip pairs
or dual lanes, chained strips or whole items, linear or affine gap) against the
oracle's maxima: alphabets around the layout rule's edge, lengths around strips
and column blocks, arbitrary integer scores with mismatches below the gap."""
import numpy as np
import pytest

from pypaswas_b200 import _native

pytestmark = pytest.mark.gpu
OFFSET = 33


def _seqs(rng, lens, letters):
    return [bytes(rng.choice(letters, int(n)).astype(np.uint8)) for n in lens]


@pytest.mark.parametrize("gap,ext", [(-5, 0), (-1, 0), (-11, -1), (-300, -7), (0, -3)])
@pytest.mark.parametrize("residues", [1, 7, 8, 20, 32, 45])
def test_every_form_gives_the_oracles_maxima(engine_lib, oracle_mod, residues, gap, ext):
    rng = np.random.default_rng(residues * 1000 - gap * 10 - ext)
    letters = np.arange(OFFSET, OFFSET + residues)
    matrix = rng.integers(-127, 40, (residues, residues)).astype(np.float32)
    np.fill_diagonal(matrix, rng.integers(1, 90, residues))
    lens = [1, 3, 4, 5, 16, 17, 24, 25, 31, 32, 33, 40, 41, 48, 49, 64, 65, 96, 97, 130]
    q = _seqs(rng, lens + rng.integers(1, 140, 20).tolist(), letters)
    t = _seqs(rng, lens + rng.integers(1, 140, 60).tolist(), letters)
    affine = ext != 0
    want = oracle_mod.pair_max(oracle_mod.OracleParams(matrix, OFFSET, gap, ext, affine, 1.0, 1.0),
                               [s.decode("latin-1") for s in q], [s.decode("latin-1") for s in t])
    e = _native.Engine(0, lib=engine_lib)
    try:
        e.set_scoring(matrix, OFFSET, gap, ext, affine, 1.0, 1.0, 1.0, float(matrix.max()), 0.2)
        e.set_queries(q, np.arange(len(q)))
        e.set_targets(t, np.arange(len(t)) + len(q))
        for dual in (1, 2):
            e.set_tuning(_native.PW_TUNE_DUAL, dual)
            for chain_min in (1, 500):
                e.set_tuning(_native.PW_TUNE_CHAIN_MIN, chain_min)
                for chain in (True, False):
                    info = e.align(score_only=True, chain=chain)
                    assert info.score_path == 0 and info.dual_lanes == (dual == 1)
                    np.testing.assert_array_equal(e.pair_max(), want)
    finally:
        e.close()
