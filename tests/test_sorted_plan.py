"""The plan of the sorted backward (``plan_sorted`` of ``csrc/msda_sorted.cu``), which is made on the host
from the call's shape alone: a small program linked to the library prints it."""

from __future__ import annotations

import pytest

from tests._host_program import host_program

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "msda_sorted.cuh"
using namespace msda_b200;
int main(int argc, char **argv) {
    for (int i = 1; i + 8 < argc; i += 9) {
        long long n[9];
        for (int j = 0; j < 9; ++j) n[j] = atoll(argv[i + j]);
        Params p{};
        const float reference = 0.f;
        p.B = n[0], p.S = n[1], p.G = (int)n[2], p.D = (int)n[3], p.Q = n[4], p.L = (int)n[5], p.K = (int)n[6];
        p.ref = n[7] ? &reference : nullptr, p.ref_coords = 2;
        SortPlan sp{};
        plan_sorted(sp, p, n[8] != 0, p.B, nullptr);
        printf("{\"pays\": %d, \"unit\": %d, \"units\": %d, \"all_runs\": %u, \"runs\": [",
               (int)sorting_pays(p, 2, n[7] != 0), sp.item_points, sp.items, sp.all_runs);
        for (int k = 0; k < kRunKinds; ++k)
            printf("%s[%u, %u, %u, %u, %d]", k ? ", " : "", sp.runs[k].run0, sp.runs[k].plane0, sp.runs[k].each,
                   sp.runs[k].unit0, sp.runs[k].log2_size);
        printf("], \"by_level\": %d, \"count_by_level\": %d, \"level_cells\": %d, \"count_cells\": %d, "
               "\"shared_cells\": %d}\n", (int)sp.scatter_by_level, (int)sp.count_by_level, sp.level_cells,
               sp.count_cells, sp.shared_cells);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    """``plans(call, ...)``: a plan per ``(B, S, G, D, Q, L, K, offsets, softmax)``."""
    return host_program(PROGRAM, tmp_path_factory.mktemp("plan"))


def _runs(plan, planes):
    """Every run as (plane, first unit, units), as the walk kernel finds them."""
    kinds = plan["runs"]
    for run in range(plan["all_runs"]):
        run0, plane0, each, unit0, log2 = kinds[sum(run >= kind[0] for kind in kinds[1:])]
        plane, nth = divmod(run - run0, each)
        yield plane0 + plane, unit0 + (nth << log2), 1 << log2


# B, S, G, D, Q, L, K, offsets, softmax
RUN_CALLS = [
    (4, 21504, 8, 32, 21504, 3, 4, 0, 0),       # many runs per warp: short ones in the last planes only
    (16, 21504, 8, 16, 21504, 3, 4, 0, 0),
    (2, 27750, 8, 32, 27750, 5, 4, 1, 1),
    (1, 20000, 1, 32, 250007, 2, 8, 0, 0),      # the same of one plane
    (8, 5376, 8, 32, 5376, 3, 4, 0, 0),
    (3, 5376, 8, 32, 5376, 3, 4, 0, 0),         # few: short ones in every plane
    (3, 11192, 6, 64, 11192, 3, 3, 1, 1),
    (16, 21504, 4, 64, 21504, 3, 4, 0, 0),      # 64 channels, many
    (2, 1344, 8, 32, 8192, 3, 8, 0, 0),         # hundreds of points per position
    (64, 300, 16, 32, 263, 2, 5, 0, 0),         # many small planes
    (1, 64, 8, 32, 32771, 1, 4, 0, 0),          # fewer runs than warps
    (1, 418, 8, 32, 24000, 2, 8, 0, 0),
    (1, 60, 2, 16, 70001, 1, 8, 0, 1),
]


def test_every_place_is_in_one_run_and_no_plane_is_cut_more_often(plans):
    """A run's ends are where sums of a plane meet in float16 once more: runs are 128 to 256 points long,
    by what a warp's share leaves room for (and longer where a pixel collects thousands), or longer, or
    made up for by longer ones of the same plane."""
    for call, plan in zip(RUN_CALLS, plans(*RUN_CALLS)):
        B, S, G, D, Q, L, K = call[:7]
        planes, points = B * G, Q * L * K
        length = min(256, max(128, planes * points // (148 * 64) // 32 * 32)) * min(16, 1 + points // S // 128)
        assert plan["unit"] * plan["units"] >= points
        taken, runs_of = set(), [0] * planes
        for plane, unit, units in _runs(plan, planes):
            runs_of[plane] += unit * plan["unit"] < points
            for u in range(unit, unit + units):
                assert u < plan["units"] and (plane, u) not in taken, (call, plane, u)
                taken.add((plane, u))
        assert len(taken) == planes * plan["units"], call
        assert max(runs_of) <= -(-points // length), call


def _cells(h, w):
    return (h + 1) * ((w + 7) // 7)


@pytest.mark.parametrize("levels", [
    [(128, 128), (64, 64), (32, 32)], [(100, 134), (50, 67), (25, 34), (13, 17)],
    [(200, 160), (100, 80), (50, 40), (25, 20)],                 # levels that halve
    [(100, 100)], [(190, 200)],                                  # all positions in one
    [(800, 20), (400, 10), (200, 5)],                            # narrow
    [(128, 128), (32, 32)], [(128, 128), (16, 16)], [(64, 64), (16, 16)], [(150, 150), (38, 38)],
    [(30, 30), (2, 2), (1, 1)],                                  # nine tenths in one
])
@pytest.mark.parametrize("K", [1, 4, 8])
def test_cells_of_ordinary_levels_are_counted_in_shared_memory(plans, levels, K):
    S, L = sum(h * w for h, w in levels), len(levels)
    finest = levels[0][0] * levels[0][1]
    for offsets in (0, 1):
        plan, = plans((2, S, 8, 32, 8 * S, L, K, offsets, offsets))
        most, plane = max(_cells(h, w) for h, w in levels), sum(_cells(h, w) for h, w in levels)
        assert (most if plan["count_by_level"] else plane) <= plan["count_cells"]
        if plan["by_level"]:
            # (what is left over is written unordered, which is as fast)
            assert most <= plan["level_cells"] or 1 < L and finest > 0.85 * S
        else:
            assert plane <= plan["shared_cells"]
