"""4-bit GEMV that keeps x in registers: full and partial last warps along K, ragged rows, against fp64."""
import pytest
import torch

from tensorplay_b200.ops.quant import quantize_weight_int4, weight_only_linear

pytestmark = pytest.mark.gpu
DEV = "cuda"


# K = 6272: 13 warps, the last with one chunk; 7552: 15 warps, the last with three; 8192: 16 full ones.
# 128, 6144 and 8320 take the form with x re-read per tile.
@pytest.mark.parametrize("K,group", [(128, 128), (6144, 128), (6272, 128), (7552, 128), (8192, 256), (8192, 128), (8320, 128)])
@pytest.mark.parametrize("N", [8, 1000, 4104])
@pytest.mark.parametrize("M,zero,bias", [(1, True, False), (5, True, True), (8, False, False), (13, True, True)])
def test_four_bit_gemv(K, group, N, M, zero, bias):
    g = torch.Generator(device=DEV)
    g.manual_seed(K + N + M)
    q, s, z = quantize_weight_int4(torch.randn(N, K, generator=g, device=DEV) * 0.02, group)
    x = (torch.randn(M, K + 16, generator=g, device=DEV) + 1).bfloat16()[:, :K]  # rows with a stride
    b = torch.randn(N, generator=g, device=DEV).bfloat16() if bias else None
    y = weight_only_linear(x, q, s, z if zero else None, b, 4, group)
    codes = torch.stack([q & 15, q >> 4], -1).reshape(N, K // group, group).double()
    zp = z.double().unsqueeze(-1) if zero else 8.0
    w = ((codes - zp) * s.double().unsqueeze(-1)).reshape(N, K)
    ref = x.double() @ w.t() + (b.double() if bias else 0.0)
    # A chunk of 128 k: two chains of eight MMAs whose partial sums stay below 143 sum |x| (128 + code, 128 + zero
    # point <= 143), each step rounded to 2^-23; then the sums over chunks and warps, of terms below 15 s sum |x|.
    sx = x.double().abs().reshape(M, K // group, group).sum(-1) @ s.double().t()
    bound = sx * (16 * 143 + 15 * (K // 128 + 4)) * 2.0 ** -23 + ref.abs() * 2.0 ** -8 + 1e-30
    assert ((y.double() - ref).abs() <= bound).all()
