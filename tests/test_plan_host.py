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


def test_planes_of_a_level_over_the_cluster(tmp_path):
    """every plane has one owner, in whole groups, and what a CTA reads of x
    lies inside the level and its ghost planes -- also a CTA that owns nothing
    because the cluster is the next power of two"""
    rows = run_plan(tmp_path, r"""
        for (int ranks : {1, 2, 4, 8, 16})
            for (int g : {1, 2})
                for (int n0 = g; n0 <= 600; n0 += g) {
                    const int P = tail_planes(n0, g, ranks), used = (n0 + P - 1) / P;
                    int launched = 1;
                    while (launched < used) launched *= 2;
                    for (int r = 0; r < launched; ++r) {
                        const Planes o = tail_own(n0, P, r), x = tail_read(o);
                        std::printf("%d %d %d %d %d %d %d %d %d %d\n", ranks, g, n0, P, launched, r, o.first, o.count,
                                    x.first, x.count);
                    }
                }
    """)
    owned, idle = {}, 0
    for row in rows:
        ranks, g, n0, P, launched, r, first, count, x0, nx = map(int, row.split())
        assert launched <= ranks and P % g == 0
        assert count % g == 0 and 0 <= count <= P
        owned.setdefault((ranks, g, n0), []).extend(range(first, first + count))
        idle += count == 0
        if nx:
            assert -1 <= x0 and x0 + nx <= n0 + 1, row
        if count:
            assert x0 <= first - 1 and x0 + nx >= first + count + 1, row
    assert idle > 0
    for (ranks, g, n0), planes in owned.items():
        assert planes == list(range(n0)), (ranks, g, n0)
