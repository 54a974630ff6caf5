"""The boundary rows of the affine band sweep (pypaswas_b200/csrc/pw_plan.h:
affine_epoch, affine_ring_rows, affine_hold), as a host model of the hand-over:
bands taken in order by a number of warps, each a step at a time in any order of
the warps, loading the row above a group of blocks ahead.  Every word that a
band accepts must come from the band above, and every band must finish."""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DRIVER = r"""
#include "pw_plan.h"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace pw;
constexpr int kGroup = 16, kSkew = 31;  // blocks a load, lanes before the storing one
struct Word { uint32_t epoch = 0; int band = -1; };
struct Band {
    int b = -1, t = 0;
    bool started = false;
    Word ahead[kGroup];
};
// nbands nblk warps rows (0: the engine's rule) held (0: no band is held back) order seed
int main(int argc, char** argv) {
    if (argc != 8) return 2;
    const int nb = atoi(argv[1]), nblk = atoi(argv[2]), warps = atoi(argv[3]);
    const int rows = atoi(argv[4]) ? atoi(argv[4]) : affine_ring_rows(nb, warps);
    const int hold = atoi(argv[5]) ? affine_hold(rows) : nb;
    const int order = atoi(argv[6]);
    std::mt19937 rng(atoi(argv[7]));
    std::vector<std::vector<Word>> ring(rows, std::vector<Word>(nblk));
    std::vector<char> finished(nb, 0);
    std::vector<Band> w(warps);
    int taken = 0, done = 0;
    long long foreign = 0, idle = 0, held = 0;
    auto load = [&](Band& B, int first) {
        for (int i = 0; i < kGroup; ++i)
            B.ahead[i] = first + i < nblk ? ring[(B.b + rows - 1) % rows][first + i] : Word{affine_epoch(B.b - 1, rows), B.b - 1};
    };
    auto act = [&](Band& B) -> bool {  // one step (or poll) of a warp's band; false: nothing moved
        if (B.b < 0) {
            if (taken == nb) return false;
            B = Band();
            B.b = taken++;
            return true;
        }
        if (!B.started) {
            if (B.b >= hold && !finished[B.b - hold]) {
                ++held;
                return false;
            }
            B.started = true;
            if (B.b > 0) load(B, 0);
            return true;
        }
        if (B.t == nblk + kSkew) {  // finishes after the band above
            if (B.b > 0 && !finished[B.b - 1]) return false;
            finished[B.b] = 1;
            ++done;
            B.b = -1;
            return true;
        }
        if (B.b > 0 && B.t % kGroup == 0) {
            for (int i = 0; i < kGroup; ++i)
                if (B.ahead[i].epoch != affine_epoch(B.b - 1, rows)) {
                    load(B, B.t);
                    return false;
                }
            for (int i = 0; i < kGroup; ++i) foreign += B.ahead[i].band != B.b - 1;
            load(B, B.t + kGroup);
        }
        const int k = B.t - kSkew;
        if (B.b + 1 < nb && k >= 0) ring[B.b % rows][k] = Word{affine_epoch(B.b, rows), B.b};
        ++B.t;
        return true;
    };
    while (done < nb && idle < 4000) {
        bool moved = false;
        for (int j = 0; j < warps; ++j) {
            // 0: a step each in turn; 1: any warp; 2: the last first; 3: any, some far ahead
            const int i = order == 0 ? j : order == 2 ? warps - 1 - j : (int)(rng() % warps);
            for (int r = order == 3 ? 1 + (int)(rng() % 40) : 1; r > 0; --r) moved = act(w[i]) || moved;
        }
        idle = moved ? 0 : idle + 1;
    }
    printf("%d %lld %lld %d\n", done == nb ? 1 : 0, foreign, held, rows);
    return 0;
}
"""


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows")
    src, exe = str(d / "rows.cpp"), str(d / "rows")
    with open(src, "w") as f:
        f.write(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(REPO, "pypaswas_b200", "csrc"), "-o", exe, src],
                   check=True)

    def run(nbands, nblk, warps, rows=0, held=1, order=0, seed=1):
        out = subprocess.run([exe] + [str(v) for v in (nbands, nblk, warps, rows, held, order, seed)],
                             capture_output=True, text=True, check=True).stdout.split()
        return dict(finished=out[0] == "1", foreign=int(out[1]), held=int(out[2]), rows=int(out[3]))
    return run


def test_model_sees_words_of_another_band(model):
    # two rows and no band held back: sound up to 127 bands, not from 128 on
    assert model(127, 75, 592, rows=2, held=0) == dict(finished=True, foreign=0, held=0, rows=2)
    for nbands in (128, 129, 141):
        assert model(nbands, 75, 592, rows=2, held=0)["foreign"] > 0


@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("nbands", [2, 125, 126, 127, 128, 129, 141, 188, 190, 252, 260])
def test_words_come_from_the_band_above(model, nbands, order):
    for nblk in (1, 16, 45, 150):
        for warps in (8, 592):
            r = model(nbands, nblk, warps, order=order, seed=nbands + nblk)
            assert r["finished"] and r["foreign"] == 0
            assert r["held"] == 0  # the engine's rows hold no band back


@pytest.mark.parametrize("order", [0, 1, 3])
@pytest.mark.parametrize("rows", [2, 3, 5])
def test_fewer_rows_hold_bands_back(model, rows, order):
    for nbands in (62 * rows + 2, 63 * rows + 1, 63 * rows + 2, 126 * rows, 400):
        r = model(nbands, 60, 592, rows=rows, order=order, seed=nbands)
        assert r["finished"] and r["foreign"] == 0


def test_rows(model):
    for nbands, warps, rows in ((1, 592, 2), (125, 592, 2), (126, 592, 3), (187, 592, 3), (188, 592, 4),
                                (700, 592, 10), (700, 64, 2)):
        assert model(nbands, 20, warps)["rows"] == rows
