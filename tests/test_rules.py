"""The host-side rules that choose a kernel's form (csrc/rules.hpp), compiled on the CPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hybrid-sparse-pde-solver_b200", "csrc")


@pytest.fixture
def evaluate(tmp_path):
    """evaluate(expressions): their values as integers, from a program that includes rules.hpp"""

    def run(exprs):
        src = tmp_path / "rules.cpp"
        exe = tmp_path / "rules"
        lines = "".join(f'    std::printf("%lld\\n", (long long)({e}));\n' for e in exprs)
        src.write_text('#include <cstdio>\n#include "rules.hpp"\nusing namespace hamlss;\n'
                       f"int main() {{\n{lines}}}\n")
        subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
        return [int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]

    return run


def test_persistent_cg_runs_only_where_its_blocks_run_together(evaluate):
    cases = [
        # cluster, blocks, active clusters, blocks an SM, SMs -> runs
        ((1, 16, 8, 0, 148), 1),
        ((1, 16, 0, 1, 148), 0),          # no GPC with that many SMs free
        ((1, 17, 8, 1, 148), 0),
        ((0, 148, 0, 1, 148), 1),
        ((0, 148, 0, 1, 147), 0),
        ((0, 148, 0, 0, 148), 0),         # not even one block an SM
        ((0, 148, 0, 2, 74), 1),
        ((0, 256, 0, 1, 300), 1),
        ((0, 257, 0, 1, 300), 0),         # more blocks than sets of partial sums
        ((0, 0, 0, 1, 148), 0),
    ]
    got = evaluate([f"persist_can_run({c[0]}, {c[1]}, {c[2]}, {c[3]}, {c[4]})" for c, _ in cases])
    assert got == [want for _, want in cases]


def test_uneven_rows_leave_the_product_tiles(evaluate):
    # 100,000 rows of 10 and some neighbouring longer ones, 32 of them a warp at most
    cases = [
        ((10, 320, 1000000), 0),
        ((100, 3200, 1003528), 0),
        ((300, 32 * 300, 1011463), 1),
        ((900, 32 * 900, 1035271), 1),
        ((900, 8 * 900, 1006996), 0),
        ((900, 900 + 31 * 10, 1000900), 0),
        ((3000, 3000, 9000000), 0),                       # a dense matrix: a row a warp
        ((900, 32 * 900, 300000000), 0),                  # hidden behind the rest of the matrix
        ((2 ** 31 - 1, 2 ** 31 - 1, 2 ** 31 - 1), 0),
    ]
    assert evaluate([f"prod_uneven({a}, {b}LL, {c}LL)" for (a, b, c), _ in cases]) == [w for _, w in cases]


def test_scattered_gathers(evaluate):
    assert evaluate([f"gathers_scattered({p}, {q})" for p, q in
                     [(0, 0), (320000, 319000), (320000, 160000), (320000, 159999), (320000, 12),
                      (8 * 65536 * 2, 8 * 65536), (1, 0), (1, 1)]]) == [0, 0, 0, 1, 1, 0, 1, 0]


def test_persistent_cg_threads(evaluate):
    assert evaluate([f"persist_threads({r}, {o})" for r, o in
                     [(256, 0), (256, 4096), (256, 4097), (256, 24000), (288, 0), (3584, 100)]]) == \
        [256, 256, 512, 512, 512, 512]


def test_sweep_kernel_by_shape(evaluate):
    ring, block, grid = evaluate([f"TriMode::{m}" for m in ("RING", "BLOCK", "GRID")])
    cases = [
        # rows, levels, entries, longest row
        ((262144, 1023, 523264, 2), ring),               # 512^2 grid
        ((262144, 1477, 523276, 14), block),             # ... with one row of 14
        ((262144, 1456, 523268, 6), ring),               # ... of 6: RING is still the better one
        ((120000, 60, 480000, 16), block),               # 4 of 16 places used, 2,000 rows a level
        ((18000, 60, 72000, 16), block),
        ((30000, 60, 480000, 16), ring),                 # all 16 used
        ((120000, 60, 240000, 8), block),                # 2 of 8 used
        ((120000, 60, 480000, 8), block),
        ((12000, 60, 24000, 8), ring),                   # narrow levels
        ((18000, 60, 36000, 8), ring),
        ((240000, 60, 1920000, 8), ring),                # all 8 used
        ((65536, 1021, 780000, 12), ring),               # 25-point stencil on 256^2
        ((49152, 765, 340000, 8), ring),                 # three unknowns a node
        ((240000, 60, 240000, 1), ring),
        ((240000, 60, 960000, 4), ring),
        ((30000, 60, 500000, 17), block),
        ((16384, 2, 32000, 2), grid),
        ((1, 1, 0, 0), ring),
        ((0, 0, 0, 0), block),
    ]
    got = evaluate([f"tri_mode({n}, {lv}, {nz}, {mr})" for (n, lv, nz, mr), _ in cases])
    assert got == [want for _, want in cases]
    assert evaluate([f"tri_places({k})" for k in (0, 1, 2, 3, 4, 5, 8, 9, 16)]) == [2, 2, 2, 4, 4, 8, 8, 16, 16]


def test_multi_dots_of_few_vectors(evaluate):
    cases = [((524287, 1), 0), ((524287, 8), 0), ((524288, 1), 1), ((524288, 8), 1), ((524288, 9), 0),
             ((4000000, 9), 0), ((1000, 1), 0)]
    assert evaluate([f"mdot_few({n}, {v})" for (n, v), _ in cases]) == [w for _, w in cases]


def test_request_footprint(evaluate):
    # device bytes that one request held at its peak on a solve lane (n, entries, restart, longest
    # row, measured on a B200 with the ring sweeps), all below the estimate
    held = [
        ((62500, 311512, 30, 18), 67.8e6),      # a grid with one row of 14 lower entries, all rows in 16 places
        ((60000, 1136184, 30, 19), 98.6e6),
        ((60000, 1136184, 5, 19), 74.6e6),
        ((64000, 1643032, 30, 27), 113.8e6),
        ((62500, 311500, 30, 5), 50.3e6),
        ((360000, 1797600, 30, 5), 289.5e6),
    ]
    got = evaluate([f"footprint_of({n}, {z}, {m}, {r})" for (n, z, m, r), _ in held])
    assert all(g >= h for g, (_, h) in zip(got, held)), got
    flat = 20 * (2 << 20) + (8 << 20)          # what an AMG setup may hold besides, whatever n is
    assert all(g <= 2 * h + flat for g, (_, h) in zip(got, held)), got
    # any size the interface takes gives a sum in range, growing with it
    big = evaluate([f"footprint_of({n}LL, {5 * n}LL, 30, 5)" for n in (10 ** 5, 10 ** 6, 10 ** 8, 2 ** 31 - 1)])
    assert big == sorted(big) and big[0] > 0 and big[3] > 1000 * (2 ** 31 - 1)
    # the batch lane's arrays, counted from their sizes (restart 1 to 32, five entries a row)
    got = evaluate([f"footprint_small(1000, 4900, {m})" for m in (1, 32)])
    for g, m in zip(got, (1, 32)):
        entries = 4 + 8 + 4 + 8 + 8 + 4        # columns, FP64, FP32, factor, level order, transpose
        rows = 4 * 4 + 4 * 8 + 4 * (2 * m + 5) + 16 + 4 + 8 + 4 + 8 + 9 * 4
        assert g >= 4900 * entries + 1000 * rows


def test_batch_groups(evaluate):
    sizes = [1, 100, 101, 200, 201, 640, 641, 1024, 1025, 4096, 4097, 16384, 16385]
    cg, gm = [0, 0, 1, 1, 2, 2, 2, 2, 3, 3, 4, 4, 5], [0, 0, 1, 1, 1, 1, 2, 2, 3, 3, 4, 4, 5]
    assert evaluate([f"batch_group({n}, true)" for n in sizes]) == cg
    assert evaluate([f"batch_group({n}, false)" for n in sizes]) == gm
    assert evaluate([f"batch_group_class({g})" for g in range(6)]) == [0, 0, 0, 1, 2, 3]
    assert evaluate([f"batch_group_width({g}, {w})" for w in (32, 128, 512) for g in (0, 1, 2, 5)]) == \
        [32, 32, 32, 32, 32, 64, 128, 128, 32, 64, 512, 512]


def test_product_tiles_stay_in_index_range(evaluate):
    # the last step's start + 512 must not pass the largest int
    assert evaluate([f"prod_indexable({k}LL)" for k in (0, 2 ** 31 - 513, 2 ** 31 - 512, 2 ** 31 - 1)]) == [1, 1, 0, 0]
