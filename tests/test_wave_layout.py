"""Sizes of the wave scratch: whatever scratch earlier frames left (waves of
`cap` paths) and whatever wave runs on it, the light subpaths that run beside
the camera rays write entries of their own inside the block, and every wave that
a scratch was made for and that is small enough runs them so.  (A preview of
4096 paths and then 1920x1080 at 24 samples, 49766400 paths in waves of
48258059, has a last wave of 1508341.)"""
import itertools
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BESIDE = 1 << 22
SIZES = sorted({1, 2, 3, 31, 255, 256, 257, 4095, 4096, 4097, 1508341, BESIDE - 1, BESIDE, BESIDE + 1, 2 * BESIDE - 1,
                2 * BESIDE, 2 * BESIDE + 1, 48258059, 2**31 - 1})

DRIVER = r"""
#include <cstdio>
#include "wave_layout.h"
int main()
{
    long long cap, wave;
    int beside, ls, ss;
    while (std::scanf("%lld %lld %d %d %d", &cap, &wave, &beside, &ls, &ss) == 5) {
        const long long q = omv::queue_entries(cap, beside != 0);
        const omv::ScratchLayout L = omv::scratch_layout(cap, q, ls, ss);
        std::printf("%lld %lld %zu %zu %zu %zu %zu\n", q, (long long)omv::light_queue_first(wave, q), L.rq0, L.rq1, L.hits,
                    L.pjob, L.bytes);
    }
}
"""


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    d = tmp_path_factory.mktemp("layout")
    (d / "driver.cpp").write_text(DRIVER)
    csrc = os.path.join(ROOT, "openmaterial-validation_gb300", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", csrc, str(d / "driver.cpp"), "-o", str(d / "driver")], check=True)

    def run(rows):
        text = "\n".join(" ".join(str(x) for x in r) for r in rows)
        out = subprocess.run([str(d / "driver")], input=text, capture_output=True, text=True, check=True).stdout
        return np.array([[int(x) for x in line.split()] for line in out.splitlines()])

    return run


@pytest.mark.parametrize("beside", [0, 1])
@pytest.mark.parametrize("slots", [(1, 1), (7, 8), (61, 62)])
def test_light_queues_lie_behind_the_wave_and_inside_the_arrays(layout, slots, beside):
    rows = [(cap, wave, beside, *slots) for cap, wave in itertools.product(SIZES, SIZES) if wave <= cap]
    for (cap, wave, *_), (q, first, rq0, rq1, hits, pjob, total) in zip(rows, layout(rows)):
        assert q >= cap
        # the arrays hold q entries each: two queues of 32 bytes, hits of 16
        assert rq0 + 32 * q <= rq1 and rq1 + 32 * q <= hits and hits + 16 * q <= pjob < total
        if first:
            assert first >= wave and first + wave <= q  # behind the camera rays' [0, wave), inside the arrays
        if beside:
            assert (first > 0) == (wave <= BESIDE)
        else:
            assert q == cap and (first > 0) == (wave <= min(BESIDE, cap // 2))


def test_second_set_costs_at_most_the_small_waves_size(layout):
    rows = [(cap, 1, 1, 7, 8) for cap in SIZES]
    for (cap, *_), (q, *_) in zip(rows, layout(rows)):
        assert q - cap == max(0, min(cap, 2 * BESIDE - cap))
