"""SwiGLU and RoPE kernels: sizes around a block's vectors, rows known only on the device, strided tokens and positions."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200.ops.rope import _rope_ref
from tensorplay_b200.parallel.moe import _swiglu_rows, _swiglu_rows_bwd

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows,I", [(1, 8), (3, 1368), (64, 64), (65, 64), (513, 24)])
def test_swiglu(rows, I):
    torch.manual_seed(rows)
    gu = (torch.randn(rows, 2 * I, device=DEV) * 3).bfloat16().requires_grad_()
    dy = torch.randn(rows, I, device=DEV).bfloat16()
    y = O.swiglu_packed(gu)
    (g,) = torch.autograd.grad(y, gu, dy)
    r = gu.detach().double().requires_grad_()
    yr = torch.nn.functional.silu(r[:, :I]) * r[:, I:]
    (gr,) = torch.autograd.grad(yr, r, dy.double())
    for a, b in ((y, yr), (g, gr)):
        assert ((a.double() - b).abs() <= 2.0 ** -8 * b.abs() + 2e-5).all()   # one rounding; fp32 arithmetic on |x| < 20
    n = torch.tensor([max(1, rows // 2)], dtype=torch.int32, device=DEV)
    assert torch.equal(_swiglu_rows(gu.detach(), n)[: n.item()], y[: n.item()])
    assert torch.equal(_swiglu_rows_bwd(dy, gu.detach(), n)[: n.item()], g[: n.item()])


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("B,T,H,D", [(1, 1, 1, 16), (2, 37, 5, 64), (3, 129, 3, 128)])
def test_rope(B, T, H, D, interleaved):
    torch.manual_seed(T)
    cos, sin = O.rope_tables(T + 50, D, 10000.0, device=DEV)
    x = torch.randn(B, T, H + 2, D, device=DEV).bfloat16()[:, :, :H]
    pos = torch.randint(0, T + 50, (B, T), device=DEV)
    for p in (None, pos):
        got = O.apply_rope(x, cos, sin, p, interleaved)
        ref = _rope_ref(x.double(), cos, sin, p, interleaved, 1.0)   # the oracle rounds to fp32 inside
        assert ((got.double() - ref.double()).abs() <= 2.0 ** -8 * ref.double().abs() + 1e-6).all()
