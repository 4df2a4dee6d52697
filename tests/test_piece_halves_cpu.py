"""Placement of the two-pass SGEMM forms' pieces in the workspace (csrc/piece_halves.h): a call may
overlap the one before only where their pieces lie apart, whatever sizes follow each other."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# workspace bytes, then the calls' piece bytes; prints lo hi apart per call
PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include "piece_halves.h"
int main(int argc, char **argv) {
    const size_t ws = strtoull(argv[1], 0, 10);
    gb::PieceRange last{0, 0, 0};
    for (int i = 2; i < argc; i++) {
        const gb::PiecePlace p = gb::place_pieces(last, strtoull(argv[i], 0, 10), ws);
        printf("%zu %zu %d\n", p.at.lo, p.at.hi, (int)p.apart);
        last = p.at;
    }
}
"""


@pytest.fixture(scope="module")
def place(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not found")
    d = tmp_path_factory.mktemp("halves")
    (d / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I",
                    os.path.join(REPO, "blas-for-multi-core-dsp_gb300", "csrc"), str(d / "t.cpp"), "-o", str(d / "t")],
                   check=True)

    def run(workspace, sizes):
        out = subprocess.run([str(d / "t"), str(workspace)] + [str(s) for s in sizes], check=True,
                             capture_output=True, text=True).stdout
        return [tuple(int(x) for x in line.split()) for line in out.splitlines()]
    return run


MB = 1 << 20


@pytest.mark.parametrize("workspace,sizes", [
    (64 * MB, [8 * MB] * 4),                              # two halves throughout
    (64 * MB, [60 * MB, MB, MB, MB]),                     # more than half, then small calls
    (64 * MB, [MB, 60 * MB, 60 * MB, MB, 40 * MB, MB, MB]),
    (64 * MB + 300, [32 * MB, 32 * MB + 256, 32 * MB, 256]),
    (1000, [512, 256, 513, 256, 256])])
def test_overlap_only_where_pieces_lie_apart(place, workspace, sizes):
    calls = place(workspace, sizes)
    last = (0, 0)
    for (lo, hi, apart), size in zip(calls, sizes):
        assert hi - lo == size and hi <= workspace
        assert not apart or hi <= last[0] or lo >= last[1]
        last = (lo, hi)


def test_calls_that_fit_a_half_alternate_and_overlap(place):
    calls = place(64 * MB, [60 * MB] + [8 * MB, 16 * MB, 32 * MB] * 2)
    assert [lo for lo, _, _ in calls] == [0] + [32 * MB, 0] * 3
    assert [apart for _, _, apart in calls] == [0, 0] + [1] * 5
