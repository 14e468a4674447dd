"""The host rules of the launches (csrc/launch_rules.h), compiled here with g++."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "wacommplusplus_b200", "csrc")


def evaluate(tmp_path, body):
    """The integers a C++ function body over the rules prints, one row per line."""
    source, exe = tmp_path / "rules.cpp", str(tmp_path / "rules")
    source.write_text('#include <cstdio>\n#include "launch_rules.h"\nusing namespace wb;\n'
                      'int main() {\n' + body + '\n}\n')
    build = subprocess.run(["g++", "-std=c++17", "-O1", "-ftrapv", str(source), "-I", CSRC, "-I",
                            os.path.join(ROOT, "include"), "-o", exe], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stderr[-500:]
    return [[int(x) for x in line.split()] for line in run.stdout.splitlines()]


# up to the largest count the entry points take: the sums stay in range and the blocks cover it
@pytest.mark.parametrize("threads", [32, 128, 256])
def test_launches_cover_every_count(tmp_path, threads):
    counts = [1, 31, 592, 593, 18944, 18945, 1 << 24, (1 << 31) - 592, (1 << 31) - 591,
              (1 << 31) - 128, (1 << 31) - 1]
    rows = evaluate(tmp_path, "".join(
        f"{{ int lanes, threads; spread_launch({n}, {threads}, lanes, threads);"
        f'printf("%d %d %d\\n", lanes, threads, launch_blocks({n}, threads / 32 * lanes)); }}\n'
        for n in counts))
    for n, (lanes, size, blocks) in zip(counts, rows):
        items = size // 32 * lanes
        assert 1 <= lanes <= 32 and size % 32 == 0 and 32 <= size <= threads
        assert (blocks - 1) * items < n <= blocks * items
        assert lanes == 32 or n <= 18944


DRAW = """
wacomm_b200_options o{}; wacomm_b200_config c{};
o.arithmetic = WACOMM_B200_ARITH_FP32; o.rng = WACOMM_B200_RNG_REFERENCE;
c.random = 1; c.trackingDirection = 1; c.dti = 30.0;
"""


# an explicit launch shape is the one that is launched: the draws ahead have a shape of their own
def test_normals_are_drawn_ahead_under_the_automatic_shape_alone(tmp_path):
    rows = evaluate(tmp_path, DRAW + """
    for (int shape = WACOMM_B200_LAUNCH_SHAPE_AUTO; shape <= 3; shape++) {
        o.launch_shape = shape;
        printf("%u\\n", draw_steps(o, c, 3600.0, 1000));
    }""")
    assert [r[0] for r in rows] == [121, 0, 0, 0, 0]


# the scratch the drop-in launcher asks for: 80 MiB, beyond 96 bytes per record, never above 1 GiB
def test_the_packed_pair_of_the_drop_in_is_bounded(tmp_path):
    mib, gib = 1 << 20, 1 << 30
    want = {(80 * mib, 1): 1, (80 * mib + 1, 1): 0, (96 * 1000000, 1000000): 1,
            (96 * 1000000, 999999): 0, (gib, 1 << 24): 1, (gib + 1, (1 << 31) - 1): 0,
            (2 * 10 ** 10, 10 ** 7): 0}
    rows = evaluate(tmp_path, "".join(f'printf("%d\\n", (int)packs_pair({b}ull, {n}ull));\n'
                                      for b, n in want))
    assert [r[0] for r in rows] == list(want.values())


# two warps per scheduler, and beyond a record per cell and level
@pytest.mark.parametrize("grid,limit", [((16, 17, 6), 37888), ((128, 128, 10), 163840),
                                        ((1 << 15, 1 << 15, 4), (1 << 31) - 1)])
def test_the_stencil_is_kept_by_thinly_spread_records(tmp_path, grid, limit):
    rows = evaluate(tmp_path, "".join(
        f'printf("%d\\n", (int)keeps_stencil({n}, {grid[0]}, {grid[1]}, {grid[2]}));\n'
        for n in (1, limit, min(limit + 1, (1 << 31) - 1))))
    assert [r[0] for r in rows] == [1, 1, int(limit == (1 << 31) - 1)]


# 16 x 17 x 6: 1,632 cells and levels; a bin more for the records that take no step
@pytest.mark.parametrize("count,forward,substeps,levels,late", [
    (1632, 0, 120, 1, 1), (1633, 0, 120, 6, 1), (1633, 1, 120, 6, 4), (400, 1, 120, 1, 4),
    (40000, 1, 120, 6, 16), (40000, 1, 4, 6, 16), (40000, 1, 3, 1, 1), (40000, 0, 1, 1, 1)])
def test_the_bins_of_the_sort(tmp_path, count, forward, substeps, levels, late):
    rows = evaluate(tmp_path, f"""
    const SortBins b = sort_bins(16, 17, 6, {count}, {forward}, {substeps});
    const SortBins most = sort_bins(16, 17, 6, {count}, {forward}, INFINITY);
    printf("%d %d %d\\n", b.levels, b.late, (int)(b.count() <= most.count()));""")
    assert rows == [[levels, late, 1]]
