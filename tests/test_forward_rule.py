"""Which forward kernel a call takes (``forward_is_wide`` of ``csrc/msda_forward.cu``), decided on the host."""

from __future__ import annotations

import pytest

from tests import test_gpu_forward_wide as wide
from tests._host_program import host_program

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "msda_common.cuh"
using namespace msda_b200;
int main(int argc, char **argv) {
    for (int i = 1; i + 7 < argc; i += 8) {
        long long n[8];
        for (int j = 0; j < 8; ++j) n[j] = atoll(argv[i + j]);
        Params p{};
        const float reference = 0.f;
        p.B = n[0], p.S = n[1], p.G = (int)n[2], p.D = (int)n[3], p.Q = n[4];
        p.ref = n[5] ? &reference : nullptr, p.ref_coords = 2;
        p.value = reinterpret_cast<const void *>(n[7]);
        const int pairs = 256 / p.D;                     // of a warp with 16 bytes per lane
        p.num_groups = (p.B * p.Q * p.G + pairs - 1) / pairs;
        printf("%d\n", (int)forward_is_wide(p, n[6] != 0));
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def is_wide(tmp_path_factory):
    """``is_wide((B, S, G, D, Q, offsets, softmax, address), ...)``."""
    return host_program(PROGRAM, tmp_path_factory.mktemp("rule"))


def test_cases_of_the_wide_forward_take_it(is_wide):
    """The comparison of the two kernels compares two kernels: aligned values take one, shifted ones the other."""
    calls = [(B, sum(h * w for h, w in levels), G, D, Q, coords != 0, softmax)
             for levels, B, Q, G, D, K, dtype, softmax, coords in wide.CASES]
    calls += [(3, 31 * 17 + 9 * 4, G, D, 6251, 0, softmax)
              for D, G, softmax in ((16, 10, 1), (32, 5, 1), (32, 5, 0), (64, 4, 1))]
    assert is_wide(*[(*call, 1 << 20) for call in calls]) == [1] * len(calls)
    assert is_wide(*[(*call, (1 << 20) + 16) for call in calls]) == [0] * len(calls)
