"""Row sums of O * dO behind the attention backward: odd lengths, strided dO and an O whose rows are not 16-byte aligned."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200.ops.attention import flash_bwd, flash_fwd

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,H", [(1, 1, 1), (2, 131, 3), (1, 300, 8)])
@pytest.mark.parametrize("shift", [0, 2])
def test_gradients_with_strided_tensors(D, B, T, H, shift):
    torch.manual_seed(T)
    q, k, v = (torch.randn(B, T, H, D, device=DEV, dtype=torch.bfloat16) for _ in range(3))
    o, lse = flash_fwd(q, k, v, True, D ** -0.5)
    do = torch.randn(B, T, 2, H, D, device=DEV, dtype=torch.bfloat16)[:, :, 1]
    moved = torch.empty(B * T * H * (D + 2) + 8, device=DEV, dtype=torch.bfloat16)
    if shift:   # rows of D + 2 elements that start 4 bytes into an aligned buffer
        o2 = moved[shift:shift + B * T * H * (D + 2)].view(B, T, H, D + 2)[..., :D]
        o2.copy_(o)
    else:
        o2 = o
    got = flash_bwd(do, q, k, v, o2, lse, True, D ** -0.5)
    O.check_status()
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    ref = torch.autograd.grad(O.attention_reference(qr, kr, vr), (qr, kr, vr), do.float())
    for g, r in zip(got, ref):
        # P, dS and the outputs rounded to bf16; a single key has a zero gradient for q and k
        assert (g.float() - r).norm().item() <= 1.5e-2 * r.norm().item() + 1e-2 * (T == 1)
