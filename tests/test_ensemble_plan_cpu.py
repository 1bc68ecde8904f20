"""How an ensemble cuts its members (physim_gb300/csrc/ensemble_plan.h), compiled
here: empty members (slots that wait for a job) are cut without a division by zero,
which some processors answer with 0 and others with a signal; a member's chunks
cover its tiles, none is empty, there are no more of them than its partial sums have
room for, and what a unit takes of them changes neither."""
from __future__ import annotations

import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "physim_gb300" / "csrc"

MAIN = r"""
#include <stdio.h>
#include "ensemble_plan.h"
int main()
{
    int n, block, chunk;
    long long even;
    while (scanf("%d %d %d %lld", &n, &block, &chunk, &even) == 4) {
        const pg::MemberCut c = pg::cut_member(n, block, chunk);
        printf("%d %d %d %d %d\n", pg::most_splits(n), c.n_jtiles, c.chunk_tiles, c.splits,
               pg::unit_chunks(c, block, even));
    }
    return 0;
}
"""


def _cuts(tmp_path, cases):
    src, exe = tmp_path / "cut.cpp", tmp_path / "cut"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], input="".join("%d %d %d %d\n" % c for c in cases), text=True,
                         capture_output=True, check=True).stdout
    return [tuple(map(int, ln.split())) for ln in out.splitlines()]


def test_cuts(tmp_path):
    sizes = [0, 1, 2, 255, 256, 257, 512, 513, 1792, 1793, 4095, 4096, 4097, 8191, 8192, 16384,
             32768, 32769, 40000, 100003, (1 << 26) - 1]
    cases = [(n, block, chunk, even) for n in sizes for block in (128, 256)
             for chunk in (4096, 8192, 16384, 65536) for even in (0, 300, 5000, 1 << 40)]
    for (n, block, chunk, even), got in zip(cases, _cuts(tmp_path, cases)):
        most, tiles, per, splits, run = got
        assert 1 <= splits <= most
        assert tiles == -(-n // block) and per >= 1
        assert splits * per >= tiles > (splits - 1) * per or n == 0
        assert per * block < chunk + block  # a chunk, rounded up to whole tiles
        assert 1 <= run <= splits and (run == 1 or run * per * block <= even)
