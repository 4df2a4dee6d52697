"""K ranges of the FP64 skinny products (csrc/split_plan.h): more ranges are taken only where the SM with the
most work does not walk more steps of K for them, whatever the tile count, K and SM count; and the planner's
longest walk is that of the kernel's own order of units."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# argv: SM count; prints how often the chosen ranges walk over 5 % more than doubled ones, by the units as the
# kernel takes them (unit u to CTA u mod grid), and how often the planner's figure is below that walk
PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include <algorithm>
#include <vector>
#include "split_plan.h"

static int64_t walk(int64_t tiles, int64_t nst, int splits, bool by_range, int sms) {
    const int64_t per = (nst + splits - 1) / splits, r = (nst + per - 1) / per;
    std::vector<int64_t> sum(sms, 0);
    for (int64_t u = 0; u < tiles * r; u++) {
        const int64_t sp = by_range ? u / tiles : u % r;
        sum[u % sms] += std::min(per, nst - sp * per);
    }
    return *std::max_element(sum.begin(), sum.end());
}

int main(int, char **argv) {
    const int sms = atoi(argv[1]);
    long long worse = 0, other = 0, out_of_range = 0;
    for (int by_range = 0; by_range < 2; by_range++)
        for (int64_t tiles = 1; tiles <= 9 * sms; tiles += tiles < 2 * sms ? 1 : 7)
            for (int64_t steps = 1; steps <= 600; steps += steps < 60 ? 1 : 37) {
                const int s = gb::oz_splits(tiles, steps, by_range, sms), d = gb::doubled_splits(tiles, steps, 2, sms);
                const int64_t chosen = walk(tiles, steps, s, by_range, sms);
                out_of_range += s < 1 || s > 64 || s > steps;
                other += gb::walked_steps(tiles, steps, s, by_range, sms) != chosen;
                worse += chosen > 1.05 * gb::walked_steps(tiles, steps, d, by_range, sms);
            }
    printf("%lld %lld %lld\n", worse, other, out_of_range);
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not found")
    d = tmp_path_factory.mktemp("splits")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I",
                    os.path.join(REPO, "blas-for-multi-core-dsp_gb300", "csrc"), str(d / "t.cpp"), "-o", str(d / "t")],
                   check=True)
    return lambda sms: subprocess.run([str(d / "t"), str(sms)], check=True, capture_output=True, text=True).stdout


@pytest.mark.parametrize("sms", [1, 3, 76, 152])
def test_more_ranges_never_walk_further(run, sms):
    assert run(sms).split() == ["0", "0", "0"]
