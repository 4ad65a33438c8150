"""GELU (tanh form) over the whole range of bf16: large and tiny inputs of both signs, forward and gradient."""
import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu


def test_tanh_form_over_the_range():
    bits = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16)
    x = bits.view(torch.bfloat16)
    x = x[torch.isfinite(x) & (x.abs() < 1e4)]
    x = x[: x.numel() // 8 * 8].cuda().requires_grad_()
    y = O.gelu(x, "tanh")
    (g,) = torch.autograd.grad(y, x, torch.ones_like(y))
    # reference through the sigmoid form, which keeps its relative precision for negative inputs
    xd = x.detach().double().requires_grad_()
    u2 = 2 * (2 / torch.pi) ** 0.5 * (xd + 0.044715 * xd ** 3)
    r = xd * torch.sigmoid(u2)
    (rg,) = torch.autograd.grad(r.sum(), xd)
    # one rounding to bf16; the exponential is good to 2 ulp of its argument (|2u| < 90 where it matters), results below
    # 1e-30 may flush
    assert ((y.double() - r).abs() <= 2.0 ** -8 * r.abs() + 1e-30).all()
    assert ((g.double() - rg).abs() <= 2.0 ** -8 * rg.abs() + 1e-5).all()
