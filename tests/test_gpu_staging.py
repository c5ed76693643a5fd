"""Shapes whose shared-memory staging lies at the size a kernel may use without opting in."""

from __future__ import annotations

import pytest
import torch

from oracle import msda_oracle as orc
from tests._abi import abi_backward, abi_forward, dev, to_np
from tests._golden import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,D", [(torch.float32, 16), (torch.bfloat16, 32)])
def test_softmax_staging_of_exactly_48_kilobytes(dtype, D):
    g = torch.Generator().manual_seed(D)
    levels, B, Q, G, K = [(7, 6), (5, 5), (4, 3), (2, 3), (1, 2)], 2, 70, 8, 3
    shapes = torch.tensor(levels)
    sizes = shapes[:, 0] * shapes[:, 1]
    starts, S, L = torch.cumsum(sizes, 0) - sizes, int(sizes.sum()), len(levels)
    v, go = dev(torch.randn(B, S, G, D, generator=g), dtype), dev(torch.randn(B, Q, G * D, generator=g), dtype)
    a = dev(torch.randn(B, Q, G, L * K, generator=g), dtype)
    l = dev(torch.rand(B, Q, G, L, K, 2, generator=g) * 1.2 - 0.1, torch.float32)
    sh, st = dev(shapes), dev(starts)
    bar = 1e-4 if dtype == torch.float32 else 1e-2
    out = abi_forward(v, sh, st, l, a, softmax=True)
    gv, _, ga = abi_backward(v, sh, st, l, a, go, softmax=True)
    ins = [t.cpu() for t in (v, sh, st, l, a)]
    e_gv, _, e_ga = orc.backward(*ins, go.cpu(), softmax=True)
    assert rel_err(to_np(out), orc.forward(*ins, softmax=True)) <= bar
    assert rel_err(to_np(gv), e_gv) <= bar and rel_err(to_np(ga), e_ga) <= bar
