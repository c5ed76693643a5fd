"""The sorted backward (``csrc/msda_sorted.cu``), which takes dense 16-bit calls of a million
points and more, against the float64 oracle where it can go wrong: strips and rows at the edges of
levels, ragged chunks of queries, every head size it has, several turns over the samples, level
tables it cannot sort, non-finite gradients."""

from __future__ import annotations

import ctypes

import pytest
import torch

from oracle import msda_oracle as orc
from tests._abi import _p, abi_backward, abi_backward_offsets, dev, dims, to_np
from tests._golden import rel_err

pytestmark = pytest.mark.gpu


def _inputs(seed, B, Q, G, D, K, levels, spread=0.3):
    g = torch.Generator().manual_seed(seed)
    shapes = torch.tensor(levels, dtype=torch.int64)
    sizes = shapes[:, 0] * shapes[:, 1]
    starts = torch.cumsum(sizes, 0) - sizes
    L, S = len(levels), int(sizes.sum())
    value = torch.randn(B, S, G, D, generator=g)
    loc = torch.rand(B, Q, G, L, K, 2, generator=g) * (1 + spread) - spread / 2
    logits = torch.randn(B, Q, G, L * K, generator=g)
    grad_out = torch.randn(B, Q, G * D, generator=g)
    return value, shapes, starts, loc, logits, grad_out


def _workspace_backward(value, shapes, starts, loc, attn, grad_out, softmax, nbytes=None):
    """``msda_b200_backward`` with the scratch it is fastest with (or ``nbytes`` of it)."""
    from deformops_b200._loader import load_library
    from deformops_b200.ops import DTYPE_CODES

    shim = load_library()
    B, S, G, D, Q, L, K = dims(value, loc)
    code = DTYPE_CODES[value.dtype]
    if nbytes is None:
        nbytes = shim.workspace_bytes(B, S, G, D, Q, L, K, code, int(softmax))
        assert nbytes > shim.scratch_bytes(B, S, G, D, Q, L, K, code), "the scratch is the plain one"
    grads = [torch.full_like(t, float("nan")) for t in (value, loc, attn)]
    scratch = torch.full((nbytes,), 0xFF, dtype=torch.uint8, device=value.device)
    st = shim.backward(_p(value), _p(shapes), _p(starts), _p(loc), _p(attn), _p(grad_out),
                       *[_p(t) for t in grads], _p(scratch), nbytes, 0, B, S, G, D, Q, L, K, code,
                       int(softmax), 1, value.device.index,
                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, shim.last_error()
    return grads


def _check(got, ins, grad_out, softmax, shapes, loc):
    truth = orc.backward(*[t.cpu() for t in ins], grad_out.cpu(), softmax=softmax)
    wh = shapes.flip(-1).double().cpu()[None, None, None, :, None, :]
    pix = loc.double().cpu() * wh - 0.5
    keep = ((pix - pix.round()).abs() >= 1e-3).all(-1, keepdim=True).numpy()
    assert rel_err(to_np(got[0]), truth[0]) <= 1e-2
    assert rel_err(to_np(got[1]) * keep, truth[1].reshape(got[1].shape) * keep) <= 1e-4
    assert rel_err(to_np(got[2]), truth[2].reshape(got[2].shape)) <= 1e-2


@pytest.mark.parametrize("dtype,softmax,D,K,levels,B,Q,G", [
    # widths that end with, one short of and one beyond a strip (W + 1 = 14, 7, 8, 22); heights 1, 2
    (torch.bfloat16, False, 32, 4, [(13, 13), (1, 6), (2, 7), (5, 21)], 1, 8209, 8),
    (torch.float16, True, 32, 5, [(11, 20), (6, 10)], 2, 6500, 8),
    (torch.bfloat16, True, 64, 3, [(9, 30), (5, 15), (3, 8)], 1, 40111, 3),
    (torch.float16, False, 64, 8, [(16, 14)], 1, 32769, 4),
    (torch.bfloat16, False, 16, 1, [(20, 20), (10, 10), (5, 5), (3, 3), (2, 2)], 3, 8333, 9),
    (torch.float16, True, 16, 64, [(12, 33), (6, 17)], 1, 2051, 4),
    # few positions: room for cells that is no multiple of eight
    (torch.bfloat16, False, 32, 4, [(8, 8)], 1, 32771, 8),
    (torch.float16, True, 64, 4, [(5, 3), (2, 2), (1, 1)], 2, 11003, 4),
    # runs of three lengths in every plane; in the last planes only
    (torch.bfloat16, False, 16, 4, [(60, 60), (30, 30)], 2, 27011, 8),
    (torch.bfloat16, True, 16, 4, [(60, 60), (30, 30)], 2, 35011, 8),
    # 12 000 positions and more are sorted a level at a time: point counts that leave threads idle, tiny
    # levels, one level, and one with more cells than a turn has room for
    (torch.bfloat16, False, 32, 3, [(110, 113), (3, 5), (1, 1)], 1, 12001, 10),
    (torch.float16, True, 16, 5, [(125, 100)], 3, 20011, 4),
    (torch.bfloat16, True, 64, 8, [(6500, 2), (10, 10)], 1, 7001, 10),
    # the largest room for a level's cells (10 122 of 10 752), larger levels first and last
    (torch.bfloat16, False, 64, 8, [(240, 290), (120, 145)], 1, 43501, 2),
    (torch.float16, True, 64, 8, [(120, 145), (240, 290)], 1, 43501, 2),
    # more cells than a CTA counts in shared memory: narrow levels
    (torch.bfloat16, False, 32, 4, [(3000, 2)], 1, 13000, 20),
])
def test_sorted_backward_matches_the_oracle(dtype, softmax, D, K, levels, B, Q, G):
    value, shapes, starts, loc, logits, grad_out = _inputs(K * D + Q, B, Q, G, D, K, levels)
    attn = logits if softmax else logits.softmax(-1)
    v, a, go = dev(value, dtype), dev(attn, dtype), dev(grad_out, dtype)
    l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
    got = _workspace_backward(v, sh, st, l, a, go, softmax)
    _check(got, (v, sh, st, l, a), go, softmax, shapes, l)


def test_samples_take_turns_when_the_scratch_holds_only_some():
    """Three samples of 4.1 M points, scratch for one and for two: the same gradients, from
    sample bases that are not 16-byte aligned in the weights (Q * G * P odd multiples of 2)."""
    from deformops_b200._loader import load_library
    from deformops_b200.ops import launch_counter

    B, Q, G, D, K, levels = 3, 45763, 5, 16, 6, [(24, 20), (7, 5), (4, 3)]
    value, shapes, starts, loc, logits, grad_out = _inputs(3, B, Q, G, D, K, levels)
    dtype = torch.bfloat16
    v, a, go = dev(value, dtype), dev(logits.softmax(-1), dtype), dev(grad_out, dtype)
    l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
    full = load_library().workspace_bytes(B, v.shape[1], G, D, Q, len(levels), K, 2, 0)
    for nbytes, turns in ((full * 45 // 100, 3), (full * 9 // 10, 2)):
        launch_counter.reset()
        got = _workspace_backward(v, sh, st, l, a, go, False, nbytes)
        assert (launch_counter.kernels, launch_counter.memsets) == (4 * turns, turns)
        _check(got, (v, sh, st, l, a), go, False, shapes, l)


@pytest.mark.parametrize("coords,offset_dtype,shape", [
    (2, torch.bfloat16, (1, 24000, 8, 32, 8, [(15, 22), (8, 11)])),        # three million points
    (4, torch.float32, (1, 24000, 8, 32, 8, [(15, 22), (8, 11)])),
    (2, torch.bfloat16, (1, 23201, 5, 64, 5, [(170, 150), (20, 30)])),     # sorted a level at a time
])
def test_sorted_backward_from_offsets(coords, offset_dtype, shape):
    """Reference points and offsets in place of locations."""
    from deformops_b200.registry import locations_from_offsets, msda, msda_from_offsets

    B, Q, G, D, K, levels = shape
    value, shapes, starts, loc, logits, grad_out = _inputs(5, B, Q, G, D, K, levels)
    dtype = torch.bfloat16
    g = torch.Generator().manual_seed(6)
    ref = torch.rand(B, Q, len(levels), coords, generator=g)
    off = dev(torch.randn(loc.shape, generator=g) * 2, offset_dtype)
    v, a, go = dev(value, dtype), dev(logits, dtype), dev(grad_out, dtype)
    r, sh, st = dev(ref, torch.float32), dev(shapes), dev(starts)
    fused = [t.clone().requires_grad_(True) for t in (v, off, a)]
    out = msda_from_offsets(fused[0], sh, st, r, fused[1], fused[2], method="softmax")
    got = torch.autograd.grad(out, fused, go)
    plain = [t.clone().requires_grad_(True) for t in (v, off, a)]
    ref_out = msda(plain[0], sh, st, locations_from_offsets(r, plain[1].float(), sh), plain[2],
                   method="softmax")
    want = torch.autograd.grad(ref_out, plain, go)
    assert torch.equal(out, ref_out)
    for x, y in zip(got, want):                     # (either is rounded to bfloat16)
        assert x.dtype == y.dtype and rel_err(to_np(x), to_np(y)) <= 1e-2


@pytest.mark.parametrize("dtype,softmax,D", [(torch.float16, False, 16), (torch.bfloat16, True, 32),
                                             (torch.float16, True, 64)])
def test_levels_that_overlap_are_served_unsorted(dtype, softmax, D):
    """Sixteen levels on the same rows ask for more cells than a plane has room for.  Thousands of
    points add to an element, so it takes the replicas of the levels to meet the bar."""
    B, Q, G, K, levels = 1, 4201, 2, 8, [(60, 1)] * 16
    value, shapes, starts, loc, logits, grad_out = _inputs(7, B, Q, G, D, K, levels)
    value, starts = value[:, :60].contiguous(), torch.zeros_like(starts)
    attn = logits if softmax else logits.softmax(-1)
    v, a, go = dev(value, dtype), dev(attn, dtype), dev(grad_out, dtype)
    l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
    got = _workspace_backward(v, sh, st, l, a, go, softmax)
    _check(got, (v, sh, st, l, a), go, softmax, shapes, l)


def test_unsorted_points_from_offsets():
    """Boxes and offsets, one NaN weight: what the direct kernels make of the same call."""
    from deformops_b200.registry import msda_from_offsets

    B, Q, G, D, K, levels = 2, 30011, 3, 64, 3, [(15, 22), (8, 11)]
    value, shapes, starts, loc, logits, grad_out = _inputs(8, B, Q, G, D, K, levels)
    g = torch.Generator().manual_seed(6)
    ref = dev(torch.rand(B, Q, len(levels), 4, generator=g) * 0.5 + 0.25)
    off = dev(torch.randn(loc.shape, generator=g), torch.float32)
    attn = logits.softmax(-1)
    attn[1, 20, 2, 4] = float("nan")
    ins = [dev(value, torch.bfloat16), off, dev(attn, torch.bfloat16)]
    sh, st, go = dev(shapes), dev(starts), dev(grad_out, torch.bfloat16)
    ins = [t.requires_grad_(True) for t in ins]
    out = msda_from_offsets(ins[0], sh, st, ref, ins[1], ins[2])
    got = torch.autograd.grad(out, ins, go)
    direct = abi_backward_offsets(ins[0].detach(), sh, st, ref, ins[1].detach(), ins[2].detach(), go)
    assert 0 < int((~torch.isfinite(got[0])).sum()) <= 4 * D
    for x, y, bar in zip(got, direct, (2e-2, 1e-4, 2e-2)):
        fine = torch.isfinite(y)
        assert torch.equal(torch.isfinite(x), fine)
        assert rel_err(to_np(x[fine]), to_np(y[fine])) <= bar


def test_non_finite_gradients_stay_in_their_corners():
    B, Q, G, D, K, levels = 1, 17000, 8, 32, 4, [(18, 16), (9, 8)]
    value, shapes, starts, loc, logits, grad_out = _inputs(9, B, Q, G, D, K, levels)
    dtype = torch.bfloat16
    grad_out[0, 11, 40] = float("inf")
    grad_out[0, 12, 200] = float("nan")
    v, a, go = dev(value, dtype), dev(logits.softmax(-1), dtype), dev(grad_out, dtype)
    l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
    got = _workspace_backward(v, sh, st, l, a, go, False)
    direct = abi_backward(v, sh, st, l, a, go)
    assert torch.equal(torch.isfinite(got[0]), torch.isfinite(direct[0]))
    for x, y in zip(got, direct):
        assert not (torch.isfinite(y) & ~torch.isfinite(x)).any()
    assert 0 < int((~torch.isfinite(got[0])).sum()) <= 2 * 2 * K * 4
    fine = torch.isfinite(got[0])
    assert rel_err(to_np(got[0][fine]), to_np(direct[0][fine])) <= 2e-2
    assert rel_err(to_np(got[1])[0, 100:], to_np(direct[1])[0, 100:]) <= 1e-5


@pytest.mark.parametrize("dtype,softmax,bad", [
    (torch.bfloat16, False, float("inf")), (torch.float16, False, float("nan")),
    (torch.bfloat16, True, float("nan")), (torch.float16, True, float("inf")),
    (torch.bfloat16, True, float("-inf")),                      # an ordinary mask: all finite
])
def test_non_finite_weights_stay_in_their_corners(dtype, softmax, bad):
    """The same elements are non-finite as on the direct path (a weight's own four corners, or its
    pair's where the softmax spreads it), and the others have the same values."""
    B, Q, G, D, K, levels = 1, 17000, 8, 32, 4, [(18, 16), (9, 8)]
    value, shapes, starts, loc, logits, grad_out = _inputs(10, B, Q, G, D, K, levels)
    loc[0, 11, 3, 0, 1] = torch.tensor([3.8 / 16, 8.1 / 18])     # its 2 x 8 window is inside the level
    attn = logits if softmax else logits.softmax(-1)
    attn[0, 11, 3, 1] = bad
    v, a, go = dev(value, dtype), dev(attn, dtype), dev(grad_out, dtype)
    l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
    got = _workspace_backward(v, sh, st, l, a, go, softmax)
    direct = abi_backward(v, sh, st, l, a, go, softmax=softmax)
    for x, y, bar in zip(got, direct, (2e-2, 1e-4, 2e-2)):
        fine = torch.isfinite(y)
        assert torch.equal(torch.isfinite(x), fine)
        assert rel_err(to_np(x[fine]), to_np(y[fine])) <= bar
    spoilt = int((~torch.isfinite(got[0])).sum())
    assert spoilt == 0 if bad == float("-inf") else 0 < spoilt <= len(levels) * K * 4 * D


@pytest.mark.parametrize("levels,overlap", [([(125, 100)], False), ([(13000, 1)] * 3, True)])
def test_unsorted_points_of_large_planes(levels, overlap):
    """What cannot be sorted, at a size that is sorted a level at a time: a NaN weight; levels on the same
    rows with more cells than a plane has room for."""
    B, Q, G, D, K = 1, 40009 // len(levels), 8, 32, 4
    value, shapes, starts, loc, logits, grad_out = _inputs(11, B, Q, G, D, K, levels)
    attn = logits.softmax(-1)
    if overlap:
        value, starts = value[:, :13000].contiguous(), torch.zeros_like(starts)
    else:
        loc[0, 11, 3, 0, 1] = torch.tensor([50.3 / 100, 60.1 / 125])
        attn[0, 11, 3, 1] = float("nan")
    dtype = torch.bfloat16
    v, a, go = dev(value, dtype), dev(attn, dtype), dev(grad_out, dtype)
    l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
    got = _workspace_backward(v, sh, st, l, a, go, False)
    direct = abi_backward(v, sh, st, l, a, go)
    for x, y, bar in zip(got, direct, (2e-2, 1e-4, 2e-2)):
        fine = torch.isfinite(y)
        assert torch.equal(torch.isfinite(x), fine)
        assert rel_err(to_np(x[fine]), to_np(y[fine])) <= bar


@pytest.mark.parametrize("levels,B,Q,K", [
    ([(40, 54), (20, 27), (10, 14), (5, 7)], 12, 2870, 4),       # short runs in the last planes only
    ([(5, 7), (10, 14), (20, 27), (40, 54)], 5, 2870, 4),        # in every plane, the finest level last
    ([(32, 32), (16, 16), (8, 8)], 2, 8192, 8),                  # runs of one length: hundreds of points a pixel
])
def test_every_plane_is_as_accurate(levels, B, Q, K):
    """The error of grad_value must not depend on where in the batch a sample stands.  What the planes
    differ in is how many sums meet in float16: no plane is cut into more than twice the runs of
    another, and rounding errors add in squares, so theirs differ by sqrt(2) at most."""
    G, D = 8, 32
    value, shapes, starts, loc, logits, grad_out = _inputs(12, B, Q, G, D, K, levels, spread=0.1)
    dtype = torch.float16
    v, a, go = dev(value, dtype), dev(logits.softmax(-1), dtype), dev(grad_out, dtype)
    l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
    got = to_np(_workspace_backward(v, sh, st, l, a, go, False)[0])
    truth = orc.backward(*[t.cpu() for t in (v, sh, st, l, a)], go.cpu(), softmax=False)[0]
    error = (((got - truth) ** 2).sum((1, 3)) / (truth ** 2).sum((1, 3))) ** 0.5
    assert error.max() <= 2 ** 0.5 * error.min(), error


def test_threads_with_different_planes_do_not_limit_each_other():
    """Calls of two pyramids from two host threads: the kernels' allowance for shared memory, which belongs
    to the device's context, must do for both whenever either is launched."""
    import threading

    from deformops_b200._loader import load_library

    shim = load_library()
    B, G, D, K = 1, 8, 16, 4
    failed = []

    def worker(levels, Q, seed):
        torch.cuda.set_device(0)
        value, shapes, starts, loc, logits, grad_out = _inputs(seed, B, Q, G, D, K, levels)
        L, S = len(levels), value.shape[1]
        v, a, go = (dev(t, torch.bfloat16) for t in (value, logits.softmax(-1), grad_out))
        l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
        grads = [torch.empty_like(t) for t in (v, l, a)]
        nbytes = shim.workspace_bytes(B, S, G, D, Q, L, K, 2, 0)
        if nbytes <= shim.scratch_bytes(B, S, G, D, Q, L, K, 2):
            failed.append("the scratch is the plain one")
        scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        torch.cuda.synchronize()
        args = (_p(v), _p(sh), _p(st), _p(l), _p(a), _p(go), *[_p(t) for t in grads], _p(scratch), nbytes,
                0, B, S, G, D, Q, L, K, 2, 0, 1, 0, ctypes.c_void_p(stream.cuda_stream))
        for _ in range(60):
            barrier.wait()          # both threads enqueue at the same time, and neither waits for the GPU
            for _ in range(50):
                if shim.backward(*args):
                    failed.append(shim.last_error())
            stream.synchronize()

    # with and without a level at a time, two sizes of each
    for small, large in (([(60, 60)], [(75, 100)]), ([(110, 110)], [(125, 125)])):
        barrier = threading.Barrier(2, timeout=60)
        threads = [threading.Thread(target=worker, args=(levels, 33000, i)) for i, levels in enumerate((small, large))]
        [t.start() for t in threads]
        [t.join() for t in threads]
    assert not failed, (len(failed), failed[0])


def test_a_pixel_that_collects_tens_of_thousands_of_points():
    """A level of one pixel beside a large one, gradients of one sign: no plane's sums may meet in float16 more often
    than runs of 256 points make them.  A sum of n equal terms, rounded as it grows, is at most n / 2 times half a
    unit off at its end."""
    levels, B, Q, G, D, K = [(125, 100), (1, 1)], 3, 20011, 5, 16, 4
    value, shapes, starts, loc, logits, grad_out = _inputs(13, B, Q, G, D, K, levels)
    dtype = torch.float16
    v, a, go = dev(value, dtype), dev(logits.softmax(-1), dtype), dev(torch.ones_like(grad_out), dtype)
    l, sh, st = dev(loc, torch.float32), dev(shapes), dev(starts)
    got = to_np(_workspace_backward(v, sh, st, l, a, go, False)[0])[:, -1]
    truth = orc.backward(*[t.cpu() for t in (v, sh, st, l, a)], go.cpu(), softmax=False)[0][:, -1]
    error = abs(got / truth - 1).max(-1)
    assert error.max() <= Q * K / 256 / 2 * 2.0 ** -12, error
