"""Listed pairs that all pass the 16-bit limit while little device memory is left:
their checkpoints, no longer shared two by two, do not fit the checkpoints' share
of the memory, and the call goes on without them; maxima and hits as with room."""
import numpy as np
import pytest

from engine_helpers import decode_hits
from pypaswas_b200 import _native

pytestmark = pytest.mark.gpu
LENGTH, QUERIES = 8000, 50  # 3.06 MB of checkpoints a pair: 153 MB two by two, 460 in the end, of 376


def _run(lib, q, t, pairs):
    e = _native.Engine(0, lib=lib)
    try:
        matrix = np.full((255, 255), -3.0, np.float32)
        np.fill_diagonal(matrix, 5.0)
        e.set_scoring(matrix, 1, -6.0, 0.0, False, 1.0, 1000.0, 1000.0, 5.0, 0.05)
        e.set_queries(q, np.arange(len(q)))
        e.set_targets(t, np.arange(len(t)) + len(q))
        e.set_pairs([a for a, _ in pairs], [b for _, b in pairs])
        info = e.align()
        return e.pair_max(), decode_hits(*e.hits()), info
    finally:
        e.close()


def test_pairs_past_the_limit_with_little_memory(engine_lib):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(2)
    bases = np.frombuffer(b"ACGT", np.uint8)
    q = [bytes(bases[rng.integers(0, 4, LENGTH)]) for _ in range(QUERIES)]
    t = [s for s in q for _ in range(2)]
    pairs = [(k // 2, k) for k in range(len(t))]
    pm, hits, info = _run(engine_lib, q, t, pairs)
    assert info.overflow_pairs == len(pairs) and info.trace_launches == 3 * info.waves
    torch.cuda.init()
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(max(free - (1 << 30), 0), dtype=torch.uint8, device="cuda")
    try:
        pm2, hits2, info2 = _run(engine_lib, q, t, pairs)
    finally:
        del held
        torch.cuda.empty_cache()
    assert info2.overflow_pairs == len(pairs) and info2.paired_cells == 0
    assert info2.trace_launches == info2.waves  # the checkpoint sweep, once a wave
    for a, b in pairs:
        assert pm[a, b] == pm2[a, b] == 5.0 * LENGTH
    assert len(hits) == len(pairs) and hits2 == hits
