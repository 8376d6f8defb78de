"""The integer arithmetic that launches and their buffers share (bmg_plan.h),
compiled by the host compiler and checked over the ranges that the kernels
take.  No GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_plan(tmp_path, body):
    """the output lines of a program whose main() is `body`"""
    gxx = shutil.which("g++")
    assert gxx, "the host compiler builds the oracle too"
    src = tmp_path / "plan.cpp"
    src.write_text('#include <cstdio>\n#include "bmg_plan.h"\nusing namespace bmg;\nint main() {\n' + body + "\n}\n")
    exe = str(tmp_path / "plan")
    subprocess.run([gxx, "-std=c++17", "-I", os.path.join(ROOT, "briscola_b200", "csrc"), "-o", exe, str(src)],
                   check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split("\n")[:-1]


def test_partial_sums_fit_their_buffer(tmp_path):
    """every reduction writes three sums a block at most: the one-cell kernels'
    grid, and that of the flexible-CG passes (16 x 16 quads a block, 64 plane
    groups, 256 on several bricks)"""
    rows = run_plan(tmp_path, r"""
        for (int nb : {1, 2, 8})
            for (int n2 : {1, 2, 3, 4, 5, 8, 12, 16, 20, 32, 48, 64, 128})
                for (int n1 : {1, 8, 16, 17, 31, 32, 33, 64, 128})
                    for (int planes : {2, 32, 64, 100, 128, 256, 300, 511, 1024}) {
                        const Level0 L{nb, n1, n2, planes, n2 % 4 == 0};
                        std::printf("%d %d %d %d %ld %ld %ld\n", nb, n2, n1, planes, cell_partials(L),
                                    step_partials(L), partials_capacity(L));
                    }
    """)
    assert len(rows) == 3 * 13 * 9 * 9
    for row in rows:
        nb, n2, n1, planes, cell, step, room = map(int, row.split())
        bx, by = (64, 4) if n2 >= 64 else (32, 8) if n2 >= 32 else (16, 16) if n2 >= 16 else (8, 32)
        assert cell == -(-n2 // bx) * -(-n1 // by) * planes
        if n2 % 4 == 0:
            assert step == -(-(n2 // 4) // 16) * -(-n1 // 16) * min(planes, 64 if nb == 1 else 256)
        else:
            assert step == cell
        assert 3 * max(cell, step) <= room, row
