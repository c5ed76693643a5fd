"""The forward with 32-byte loads per lane (dense calls of 16-bit values), against the float64 oracle.

The sizes are those its rule sends there (two queries or more per four positions; 16 channels and some
ten thousand pairs, or enough rounds of its warps), with point counts that leave the last turn of a slot
partly empty, pair counts that leave the last warp so, and a value tensor that is not 32-byte aligned,
which takes the other kernel and has to give the same bits.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import msda_oracle as orc
from tests._abi import abi_forward, abi_forward_offsets, dev, to_np
from tests._golden import rel_err

pytestmark = pytest.mark.gpu

# levels, B, Q, G, D, K, dtype, softmax, reference coordinates (0: locations; below 0: offsets in float32)
CASES = [
    ([(19, 23), (5, 7), (1, 1)], 3, 1001, 4, 16, 1, torch.float16, False, 0),      # 3 points, 1 lane a slot
    ([(19, 23), (5, 7)], 3, 1001, 4, 16, 3, torch.bfloat16, True, 2),              # 6 points, two a lane
    ([(31, 17)], 3, 6251, 5, 32, 2, torch.bfloat16, False, 0),                    # fewer points than a turn
    ([(31, 17), (9, 4), (3, 2)], 3, 6251, 5, 32, 2, torch.float16, True, 4),      # 6: half a last turn
    ([(31, 17), (9, 4), (3, 2)], 3, 6251, 5, 32, 3, torch.bfloat16, False, 0),    # 9: one point a lane
    ([(40, 30), (7, 1)], 1, 33337, 3, 64, 3, torch.float16, False, 0),             # 6 points, slots of four
    ([(40, 30), (7, 1)], 1, 33337, 3, 64, 4, torch.bfloat16, True, 2),
    ([(12, 50)], 2, 12345, 2, 128, 5, torch.bfloat16, False, 0),                   # 5 points, slots of eight
    # offsets divided by sizes that have no exact reciprocal: the other kernel divides
    ([(49, 33), (1021, 3), (11, 107), (7, 1)], 3, 6251, 5, 32, 2, torch.float16, False, 2),
    ([(83, 41), (3, 347), (25, 13)], 2, 12501, 3, 64, 1, torch.float16, True, 2),
    # two points a lane in one load: locations; float32 offsets
    ([(19, 23), (5, 7)], 3, 1001, 4, 16, 2, torch.float16, False, 0),
    ([(19, 23), (5, 7)], 3, 1001, 4, 16, 3, torch.bfloat16, True, 0),
    ([(19, 23), (5, 7)], 3, 1001, 4, 16, 2, torch.float16, True, -2),
    ([(31, 17), (9, 4), (3, 2)], 3, 6251, 5, 32, 2, torch.bfloat16, False, -4),
    ([(12, 50), (6, 25)], 2, 12345, 3, 128, 5, torch.float16, True, 2),           # slots of eight, 10 points
    ([(12, 50), (6, 25)], 2, 12345, 3, 128, 3, torch.bfloat16, True, -2),
]


@pytest.mark.parametrize("levels,B,Q,G,D,K,dtype,softmax,coords", CASES)
def test_wide_forward_matches_the_oracle(levels, B, Q, G, D, K, dtype, softmax, coords):
    gen = torch.Generator().manual_seed(7)
    shapes = np.array(levels, dtype=np.int64)
    sizes = shapes.prod(1)
    starts = np.cumsum(sizes) - sizes
    S, L = int(sizes.sum()), len(levels)
    value = torch.randn(B, S, G, D, generator=gen).to(dtype)
    attn = torch.randn(B, Q, G, L * K, generator=gen)
    attn = (attn if softmax else torch.softmax(attn, -1)).to(dtype)
    sh, st = dev(shapes), dev(starts)
    wh = torch.tensor(shapes[:, ::-1].copy(), dtype=torch.float32).view(1, 1, 1, L, 1, 2)
    if coords:
        offsets = (2 * torch.randn(B, Q, G, L, K, 2, generator=gen)).to(dtype if coords > 0 else torch.float32)
        coords = abs(coords)
        ref = torch.rand(B, Q, L, coords, generator=gen)
        r = ref.view(B, Q, 1, L, 1, coords)
        loc = (r + offsets.float() / wh if coords == 2
               else r[..., :2] + offsets.float() / K * r[..., 2:] * 0.5)
        run = lambda v: abi_forward_offsets(v, sh, st, dev(ref), dev(offsets), dev(attn), softmax=softmax)
    else:
        loc = 1.6 * torch.rand(B, Q, G, L, K, 2, generator=gen) - 0.3
        loc[:, ::7, :, 0, 0] = float("nan")
        run = lambda v: abi_forward(v, sh, st, dev(loc), dev(attn), softmax=softmax)
    v = dev(value)
    assert v.data_ptr() % 32 == 0
    shifted = torch.empty(v.numel() + 8, dtype=dtype, device="cuda")[8:].view(v.shape)
    shifted.copy_(v)
    assert shifted.data_ptr() % 32 == 16
    out, other = to_np(run(v)), to_np(run(shifted))
    want = orc.forward(value, shapes, starts, loc, attn, softmax=softmax, precision="f64")
    # half a unit of the 16-bit result in the last place of its largest element, and as much again
    # for float32 sums of L * K * 4 terms
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert rel_err(out, want) < 2 * unit
    # the two kernels add the same products in the same order
    assert np.array_equal(out, other)


@pytest.mark.parametrize("D,softmax,dtype", [(16, True, torch.bfloat16), (32, True, torch.float16),
                                             (32, False, torch.bfloat16), (64, True, torch.bfloat16)])
def test_non_finite_operands_give_what_the_other_kernel_gives(D, softmax, dtype):
    """Infinities and NaN in the values, in weights and logits, and rows of nothing but -inf logits."""
    levels, B, Q, K = [(31, 17), (9, 4)], 3, 6251, 2
    G, S, L = {16: 10, 32: 5, 64: 4}[D], 31 * 17 + 9 * 4, 2
    gen = torch.Generator().manual_seed(8)
    shapes = np.array(levels, dtype=np.int64)
    sh, st = dev(shapes), dev(np.array([0, 31 * 17]))
    value = torch.randn(B, S, G, D, generator=gen)
    value[0, 5::97, 0, 3] = float("inf")
    value[1, 7::89, -1, 0] = float("-inf")
    value[2, 11::83, :, D - 1] = float("nan")
    attn = torch.randn(B, Q, G, L * K, generator=gen)
    attn = attn if softmax else torch.softmax(attn, -1)
    attn[:, ::13, 0, 1] = float("-inf") if softmax else float("inf")
    attn[:, ::17, 1] = float("-inf") if softmax else 0.0
    attn[:, ::101, 1, 0] = float("nan")
    loc = 1.2 * torch.rand(B, Q, G, L, K, 2, generator=gen) - 0.1
    value, attn = value.to(dtype), attn.to(dtype)
    v, a, l = dev(value), dev(attn), dev(loc)
    shifted = torch.empty(v.numel() + 8, dtype=dtype, device="cuda")[8:].view(v.shape)
    shifted.copy_(v)
    assert v.data_ptr() % 32 == 0 and shifted.data_ptr() % 32 == 16
    out = to_np(abi_forward(v, sh, st, l, a, softmax=softmax))
    other = to_np(abi_forward(shifted, sh, st, l, a, softmax=softmax))
    assert np.array_equal(out, other, equal_nan=True)
    want = orc.forward(value, shapes, np.array([0, 31 * 17]), loc, attn, softmax=softmax, precision="f64")
    # (a corner outside its level has weight zero and is read at the border: 0 * inf is NaN there, where
    # the oracle leaves it out; the other way round nothing may be lost)
    assert not (np.isfinite(out) & ~np.isfinite(want)).any()
    fine = np.isfinite(out)
    assert 0.5 < fine.mean() < 1.0
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert rel_err(out[fine], want[fine]) < 2 * unit
