"""The projections of the layers: column sums (``csrc/msda_linear.cu``) and the autograd path around
them (``core/linear.py``) against torch."""

from __future__ import annotations

import ctypes

import pytest
import torch
from torch import nn

from deformops_b200.core.linear import project, project_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,cols,shift", [(0, 8, 0), (1, 1, 0), (31, 7, 0), (32, 54, 0), (2049, 96, 0),
                                             (4099, 256, 0), (2048, 257, 0), (3000, 264, 4), (65, 1032, 0)])
def test_column_sums(dtype, rows, cols, shift):
    """Row counts around a CTA's, columns around a block's, rows that are not 16-byte aligned."""
    from deformops_b200._loader import load_library
    from deformops_b200.ops import DTYPE_CODES

    shim = load_library()
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows * cols + shift, generator=g, device="cuda").to(dtype)[shift:].view(rows, cols)
    out = torch.full((cols,), float("nan"), dtype=dtype, device="cuda")
    scratch = torch.full((shim.column_sums_scratch_bytes(rows, cols),), 0xFF, dtype=torch.uint8, device="cuda")
    p = [ctypes.c_void_p(t.data_ptr()) for t in (x, out, scratch)]
    if rows == 0:
        p[0] = p[1]                              # (an empty tensor has no address)
    st = shim.column_sums(*p, rows, cols, DTYPE_CODES[dtype],
                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, shim.last_error()
    want = x.double().sum(0)
    eps = {torch.float32: 1e-6, torch.float16: 1e-3, torch.bfloat16: 8e-3}[dtype]
    assert torch.allclose(out.double(), want, rtol=eps, atol=eps * max(rows, 1) ** 0.5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_projections_match_the_modules(dtype):
    torch.manual_seed(0)
    a, b = nn.Linear(40, 54).to("cuda", dtype), nn.Linear(40, 27).to("cuda", dtype)
    x = torch.randn(3, 800, 40, device="cuda", dtype=dtype)
    ga, gb = torch.randn(3, 800, 54, device="cuda", dtype=dtype), torch.randn(3, 800, 27, device="cuda", dtype=dtype)
    bar = 1e-5 if dtype == torch.float32 else 1e-2

    def grads(pair):
        xs = x.clone().requires_grad_(True)
        out = pair(xs)
        wanted = [xs, a.weight, a.bias, b.weight, b.bias]
        return [*out, *torch.autograd.grad(list(out), wanted, [ga, gb])]

    got, want = grads(lambda t: project_pair(a, b, t)), grads(lambda t: (a(t), b(t)))
    assert "LinearFunction" in project(a, x).grad_fn.name() and "LinearFunction" in got[0].grad_fn.name()
    for u, v in zip(got, want):
        assert u.dtype == v.dtype and u.shape == v.shape
        assert float((u.double() - v.double()).norm() / v.double().norm()) < bar
    # one output unused; a frozen weight; a hook (the module itself is called)
    xs = x.clone().requires_grad_(True)
    only_b = torch.autograd.grad(project_pair(a, b, xs)[1], [xs, b.bias], gb)
    ref_b = torch.autograd.grad(b(xs), [xs, b.bias], gb)
    assert all(torch.allclose(u.float(), v.float(), rtol=bar, atol=bar * 30) for u, v in zip(only_b, ref_b))
    a.weight.requires_grad_(False)
    project(a, x).backward(ga)
    assert a.weight.grad is None and a.bias.grad is not None
    a.register_forward_hook(lambda m, i, o: o * 0)
    assert not project(a, x).any()


def test_projection_gradients_can_be_differentiated():
    torch.manual_seed(1)
    a = nn.Linear(8, 4).cuda()
    x = torch.randn(2500, 8, device="cuda", requires_grad=True)

    def second(f):
        y = f(x)
        (gx,) = torch.autograd.grad(y.square().sum(), x, create_graph=True)
        return torch.autograd.grad(gx.square().sum(), [x, a.weight, a.bias])

    for u, v in zip(second(lambda t: project(a, t)), second(a)):
        assert torch.allclose(u, v, rtol=1e-4, atol=1e-3)
