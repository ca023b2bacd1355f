"""The host rules of csrc/tiles.h, compiled on their own (no GPU)."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2_b200", "csrc")


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    """rule(expression): the integer value of a C++ expression over tiles.h."""
    d = tmp_path_factory.mktemp("tiles")

    def run(*expr):
        src = d / "t.cpp"
        src.write_text('#include <cstdio>\n#include "tiles.h"\nusing namespace mm;\nint main() {\n'
                       + "".join('std::printf("%%lld\\n", (long long)(%s));\n' % e for e in expr) + "}\n")
        subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(d / "t")], check=True)
        return [int(v) for v in subprocess.run([str(d / "t")], check=True, capture_output=True, text=True).stdout.split()]
    return run


def test_columns_use_the_sms_of_narrow_films(rule):
    """Narrow films take at least 60 blocks where they have the columns, and never more than one
    block per SM by halving below four columns; wide ones keep rows of 32 bytes."""
    line = {n1: 3 * 2 * n1 * 8 for n1 in (600, 1000, 1200, 2048)}
    got = rule(*["col_tiles(%d, %d, 1).tc" % (line[n1], cols) for n1 in line for cols in (65, 129, 257, 1025)])
    assert got == [1, 1, 2, 4, 1, 1, 2, 4, 1, 1, 2, 2, 1, 1, 2, 2]
    # short lines keep four columns; the tile never passes 200 KB
    assert rule("col_tiles(1536, 25, 6).tc", "col_tiles(98304, 65, 64).tc") == [4, 2]


def test_column_threads(rule):
    """512 where a block has its SM to itself."""
    assert rule("col_tiles(28800, 1025, 1).threads", "col_tiles(30720, 1025, 1).threads",
                "col_tiles(28800, 513, 1).threads", "col_tiles(1536, 97, 24).threads") == [256, 512, 512, 256]


def test_split_columns(rule):
    assert rule("split_columns(65, 1)", "split_columns(257, 1)", "split_columns(513, 1)", "split_columns(65, 8)") == \
        [2, 2, 4, 4]


def test_few_long_columns_take_their_own_stages(rule):
    assert rule("line_columns(2048, 198)", "line_columns(2048, 390)", "line_columns(4096, 102)",
                "line_columns(4096, 198)", "line_columns(1024, 8)", "line_columns(1200, 8)") == [1, 0, 1, 0, 0, 0]
    assert rule("line_multiply(4096, 129)", "line_multiply(4096, 257)", "line_multiply(2048, 65)",
                "line_multiply(3000, 9)") == [1, 0, 1, 0]


def test_small_weight_gradients_stage_each_tap(rule):
    small = [(1, 1), (5, 1), (81, 1), (162, 1), (81, 4), (18, 16), (10, 48), (9, 48)]
    large = [(289, 1), (133, 3), (81, 12), (67, 16), (21, 48), (4225, 64)]
    assert rule(*["wgrad_by_ring(%d, %d)" % v for v in small]) == [0] * len(small)
    assert rule(*["wgrad_by_ring(%d, %d)" % v for v in large]) == [1] * len(large)


@pytest.mark.parametrize("full,row_threads", [(16, 24), (8, 48), (4, 96)])
def test_row_tiles_of_small_grids_run_in_one_wave(rule, full, row_threads):
    """Fewer full tiles than SMs: every row is covered, a block has 32 to 384 threads and enough of
    them for its row transforms, and no block waits for another to end."""
    cases = [(rows, n2, nsim, fit) for rows in (1, 37, 147, 149, 150, 296, 297, 450, 512, 590) for n2 in (8, 100, 256, 1024)
             for nsim in (1, 3) for fit in (416, 800, 1152) if (rows + full - 1) // full * nsim < 148]
    got = rule(*["row_tile(%d, %d, %d, %d, %d, 0, %d).%s" % (full, row_threads, r, n, s, f, k)
                 for r, n, s, f in cases for k in ("rpb", "threads")])
    for (rows, n2, nsim, fit), rpb, threads in zip(cases, got[::2], got[1::2]):
        assert 1 <= rpb <= full and 32 <= threads <= 384 and threads % 32 == 0 and threads >= rpb * row_threads
        assert -(-rows // rpb) * nsim <= 148 * max(1, fit // threads)


def test_multiply_tiles_stay_apart(rule):
    """Narrowed columns of small films still halve and double by the plan's tile."""
    assert rule(*["colmul4_shift(64, 8, 257, %d)" % t for t in (-1, 0, 1)]) == [-3, -3, -2]
    assert rule(*["colmul4_shift(64, 8, 513, %d)" % t for t in (-1, 0, 1)]) == [-3, -2, -1]
    assert rule(*["colmul4_shift(64, 8, 100000, %d)" % t for t in (-1, 0, 1)]) == [-1, 0, 1]
    assert rule(*["colmul4_shift(256, 16, 129, %d)" % t for t in (-1, 0, 1)]) == [-1, 0, 1]
