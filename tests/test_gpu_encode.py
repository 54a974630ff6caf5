"""Sequence sets encoded on the device: lengths around the 16-byte chunks, empty
records, sorted and unsorted, sets on either side of the size that goes to the
device by itself; invalid residues are reported from both."""
import numpy as np
import pytest

import cases
from engine_helpers import configure
from pypaswas_b200 import _native, scores
from pypaswas_b200.exceptions import InvalidOptionException

pytestmark = pytest.mark.gpu


def _set(rng, residues, order):
    lens = [0, 1, 15, 16, 17, 31, 32, 33, 48]
    while sum(lens) < residues:
        lens.append(int(rng.integers(0, 400)))
    lens[-1] -= sum(lens) - residues
    lens = np.array(lens)
    if order == "sorted":
        lens = -np.sort(-lens)
    return [bytes(rng.choice(np.frombuffer(b"ACGTNacgt", np.uint8), int(n))) for n in lens]


@pytest.mark.parametrize("residues", [3000, (1 << 18) - 1, 1 << 18, (1 << 18) + 5])
@pytest.mark.parametrize("order", ["sorted", "unsorted"])
def test_either_side_of_the_direct_size(engine_lib, oracle_mod, residues, order):
    rng = np.random.default_rng(residues)
    big, small = _set(rng, residues, order), _set(rng, 300, order)
    st = cases.Settings(minimum_score="6")
    score = scores.make_score(st)
    p = cases.oracle_params(oracle_mod, score)
    e = _native.Engine(0, lib=engine_lib)
    try:
        configure(e, score, st)
        for q, t in ((big, small), (small, big)):
            e.set_queries(q, np.arange(len(q)))
            e.set_targets(t, np.arange(len(t)) + len(q))
            e.align(score_only=True)
            np.testing.assert_array_equal(e.pair_max(), oracle_mod.pair_max(
                p, [s.decode().upper() for s in q], [s.decode().upper() for s in t]))
        bad = list(big)
        bad[-1 if order == "unsorted" else 0] = b"AC-GT"
        for q, t, what in ((bad, small, "query"), (small, bad, "target")):
            e.set_queries(q, np.arange(len(q)))
            e.set_targets(t, np.arange(len(t)) + len(q))
            with pytest.raises(InvalidOptionException, match=what + " residue outside the scoring matrix: code 45"):
                e.align(score_only=True)
    finally:
        e.close()
