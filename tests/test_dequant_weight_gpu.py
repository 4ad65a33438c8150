"""Dequantised weights, bit for bit: groups that are and are not powers of two, ragged sizes, zero points and none."""
import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("bits,N,K,group", [(4, 3, 128, 128), (4, 129, 1032, 24), (4, 1000, 4096, 32), (8, 1, 8, 0),
                                            (8, 77, 264, 0), (8, 515, 2048, 64), (8, 33, 1040, 104)])
def test_matches_formula(bits, N, K, group):
    torch.manual_seed(N)
    g = group or K
    q = torch.randint(0, 256, (N, K if bits == 8 else K // 2), device=DEV, dtype=torch.uint8)
    scale = (torch.rand(N, K // g, device=DEV) + 0.01).bfloat16()
    for zero in ([None, torch.rand(N, K // g, device=DEV).mul(15).bfloat16()] if bits == 4 else [None]):
        if bits == 4:
            code = torch.stack((q & 0xF, q >> 4), -1).reshape(N, K // g, g).float()
            ref = (code - (8.0 if zero is None else zero.float().unsqueeze(-1))) * scale.float().unsqueeze(-1)
        else:
            ref = q.view(torch.int8).float().view(N, K // g, g) * scale.float().unsqueeze(-1)
        got = O.dequantize_weight(q if bits == 4 else q.view(torch.int8), scale, zero, bits, group)
        assert torch.equal(got, ref.reshape(N, K).bfloat16())
