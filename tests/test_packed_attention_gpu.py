"""Attention over a packed projection without rotation: values and gradient against the slices of the projection."""
import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("B,T,Hq,Hkv,D", [(2, 130, 4, 4, 64), (1, 257, 4, 2, 128), (3, 1, 2, 2, 64), (2, 40, 2, 2, 32)])
def test_packed_without_rotation(B, T, Hq, Hkv, D):
    torch.manual_seed(T)
    qkv = torch.randn(B, T, (Hq + 2 * Hkv) * D, device=DEV).bfloat16().requires_grad_()
    do = torch.randn(B, T, Hq * D, device=DEV).bfloat16()
    o = O.qkv_attention(qkv, None, None, None, Hq, Hkv, D)
    (g,) = torch.autograd.grad(o, qkv, do)
    p = qkv.view(B, T, Hq + 2 * Hkv, D)
    r = O.flash_attention(p[:, :, :Hq], p[:, :, Hq:Hq + Hkv], p[:, :, Hq + Hkv:])
    (rg,) = torch.autograd.grad(r, qkv, do.view(r.shape))
    O.check_status()
    assert torch.equal(o, r.reshape(o.shape))   # the same kernels on the same memory
    assert torch.equal(g, rg)
