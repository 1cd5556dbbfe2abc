"""The count at a grid barrier's crossings (csrc/hzb_tally.h), played through on
the CPU with CTAs that read late."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "hazmath_b200", "csrc")
SHIM = r"""
#include "hzb_tally.h"
#include <vector>
// Steps of the CTAs in the given order: a CTA arrives, then polls until its
// crossing is complete; totals[c * rounds + r]: what it found.
extern "C" long long play(int ctas, int rounds, const int *counts, long long steps,
                          const int *order, long long *totals) {
    std::vector<hzb::GridTally> T(ctas);
    std::vector<int> round(ctas, 0), waits(ctas, 0);
    unsigned long long words[2] = {0, 0};
    for (long long k = 0; k < steps; ++k) {
        const int c = order[k];
        if (round[c] == rounds) continue;
        if (!waits[c]) {
            ++T[c].r;
            words[T[c].word()] += hzb::GridTally::arrival((unsigned)counts[c * rounds + round[c]]);
            waits[c] = 1;
        } else if (T[c].complete(words[T[c].word()], (unsigned)ctas)) {
            totals[c * rounds + round[c]++] = T[c].total(words[T[c].word()]);
            waits[c] = 0;
        }
    }
    long long left = 0;
    for (int c = 0; c < ctas; ++c) left += rounds - round[c];
    return left;
}
"""


@pytest.fixture(scope="module")
def play(tmp_path_factory):
    d = tmp_path_factory.mktemp("tally")
    src, so = str(d / "shim.cpp"), str(d / "shim.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, src, "-o", so],
                   check=True)
    lib = C.CDLL(so)
    lib.play.restype = C.c_longlong

    def run(counts, order):
        counts = np.ascontiguousarray(counts, np.int32)
        order = np.ascontiguousarray(order, np.int32)
        ctas, rounds = counts.shape
        totals = np.full((ctas, rounds), -1, np.int64)
        ip = lambda a: a.ctypes.data_as(C.c_void_p)
        left = lib.play(ctas, rounds, ip(counts), C.c_longlong(len(order)), ip(order), ip(totals))
        return left, totals
    return run


def test_a_late_reader_sees_no_later_counts(play):
    # CTA 1 completes crossing 1, arrives at 2 with a count, and only then CTA 0
    # reads crossing 1
    counts = [[1, 0, 0], [0, 1, 0]]
    left, totals = play(counts, [0, 1, 1, 1, 0, 0, 0, 1, 1, 1, 0, 0, 1, 0])
    assert left == 0
    assert np.array_equal(totals, [[1, 2, 2], [1, 2, 2]])


@pytest.mark.parametrize("ctas", [1, 2, 3, 148])
def test_every_cta_finds_the_same_totals(play, ctas):
    rng = np.random.default_rng(ctas)
    rounds = 60
    counts = rng.integers(0, 3, (ctas, rounds)) * (rng.random((ctas, rounds)) < 0.2)
    want = np.cumsum(counts.sum(0))
    for trial in range(20):
        # runs of steps by one CTA, so that others read late
        order = np.repeat(rng.integers(0, ctas, 4000 * ctas), rng.integers(1, 5, 4000 * ctas))
        left, totals = play(counts, order)
        assert left == 0
        assert np.array_equal(totals, np.broadcast_to(want, totals.shape))
