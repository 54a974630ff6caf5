"""The queue of a band sweep (pypaswas_b200/csrc/pw_plan.h, plan_band_queue),
compiled on the host: every band of every pair is queued once, after the band
above it -- short pairs beside very long ones too."""
import os
import subprocess

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DRIVER = r"""
#include "pw_plan.h"
#include <cstdio>
int main() {
    int n, warps, lead;
    if (scanf("%d %d %d", &n, &warps, &lead) != 3) return 2;
    std::vector<int> nb(n); std::vector<int64_t> st(n);
    for (int k = 0; k < n; ++k) { long long a; if (scanf("%d %lld", &nb[k], &a) != 2) return 2; st[k] = a; }
    std::vector<pw::PlanEntry> q;
    pw::plan_band_queue(nb, st, warps, lead, q);
    for (auto& e : q) printf("%d %d %d\n", e.item, e.strip, e.pred);
    return 0;
}
"""


@pytest.fixture(scope="module")
def queue(tmp_path_factory):
    d = tmp_path_factory.mktemp("queue")
    src, exe = str(d / "queue.cpp"), str(d / "queue")
    with open(src, "w") as f:
        f.write(DRIVER)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(REPO, "pypaswas_b200", "csrc"), "-o", exe, src],
                   check=True)

    def run(nbands, steps, warps, lead=48):
        inp = "%d %d %d\n" % (len(nbands), warps, lead) + "".join("%d %d\n" % v for v in zip(nbands, steps))
        out = subprocess.run([exe], input=inp, capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, ln.split())) for ln in out.splitlines()]
    return run


@pytest.mark.parametrize("nbands,steps,warps", [
    ([1563, 2], [25031, 32], 592),               # 100 kb x 400 kb beside a short pair of 300 rows
    ([4000, 3, 1, 2], [250031, 40, 33, 32], 592),
    ([3, 2, 1], [100, 90, 80], 592),
    ([1], [31], 592),
    ([5, 5, 4, 4, 3, 3, 2, 2, 1, 1], [400] * 10, 16),  # band-major order
    ([900] + [2] * 200, [60000] + [40] * 200, 1184),
])
def test_every_band_is_queued_after_the_band_above(queue, nbands, steps, warps):
    q = queue(nbands, steps, warps)
    assert len(q) == sum(nbands)
    at = {}
    for k, (pair, band, pred) in enumerate(q):
        assert (pair, band) not in at
        at[pair, band] = k
        assert pred == (at[pair, band - 1] if band else -1)
    assert set(at) == {(p, b) for p, n in enumerate(nbands) for b in range(n)}


def test_random_pairs(queue):
    rng = np.random.default_rng(4)
    for _ in range(20):
        n = int(rng.integers(1, 60))
        nb = np.maximum(1, (10 ** rng.uniform(0, 3.5, n)).astype(int)).tolist()
        st = (31 + 10 ** rng.uniform(0, 5, n)).astype(int).tolist()
        pairs = sorted(zip(nb, st), key=lambda v: -v[0] * v[1])
        q = queue([a for a, _ in pairs], [b for _, b in pairs], int(rng.integers(1, 2400)))
        assert sorted((p, b) for p, b, _ in q) == [(p, b) for p, (k, _) in enumerate(pairs) for b in range(k)]
