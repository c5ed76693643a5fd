"""The 16-bit backward in one launch (small calls whose scratch has room for it), against
the float64 oracle: a single CTA, replicas of a coarse level, several sets of groups per CTA."""

from __future__ import annotations

import pytest
import torch

from tests._abi import dev, to_np
from tests._golden import rel_err
from tests.test_gpu_sorted import _check, _inputs, _workspace_backward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("softmax,D,K,levels,B,Q,G", [
    (False, 32, 1, [(3, 2)], 1, 1, 1),
    (True, 32, 4, [(9, 7), (2, 2)], 2, 700, 8),
    (False, 8, 2, [(20, 17), (5, 4)], 3, 5400, 4),
    (True, 64, 3, [(13, 9)], 1, 4000, 20),
])
def test_one_launch_backward_matches_the_oracle(dtype, softmax, D, K, levels, B, Q, G):
    value, shapes, starts, loc, logits, grad_out = _inputs(Q, B, Q, G, D, K, levels)
    v, go = dev(value, dtype), dev(grad_out, dtype)
    a = dev(logits if softmax else logits.softmax(-1), dtype)
    l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
    got = _workspace_backward(v, sh, st, l, a, go, softmax)
    _check(got, (v, sh, st, l, a), go, softmax, shapes, l)


def test_one_launch_backward_runs_beside_another_streams_kernel():
    """It takes the room that there is: a kernel that stays on one SM does not hold it up."""
    dtype = torch.float16
    value, shapes, starts, loc, logits, grad_out = _inputs(1, 4, 300, 8, 32, 4, [(50, 67), (25, 34)])
    v, a, go = dev(value, dtype), dev(logits.softmax(-1), dtype), dev(grad_out, dtype)
    l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
    want = _workspace_backward(v, sh, st, l, a, go, False)        # (the kernel is loaded, the scratch cached)
    torch.cuda.synchronize()
    side, main = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(400_000_000)                            # one thread, about 0.2 s
        left = side.record_event()
    with torch.cuda.stream(main):
        got = _workspace_backward(v, sh, st, l, a, go, False)
    main.synchronize()
    assert not left.query(), "the call waited for the other stream"
    side.synchronize()
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    assert rel_err(to_np(got[0]), to_np(want[0])) <= 1e-2
