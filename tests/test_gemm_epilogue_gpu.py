"""Bias in the GEMM epilogues: vector loads, and the scalar form for fp32, unaligned and last columns."""
import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("impl", ["pair", "single"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N", [(256, 256), (130, 264), (300, 520), (1, 40)])
@pytest.mark.parametrize("shift", [0, 1])
def test_bias_columns(impl, dtype, M, N, shift):
    torch.manual_seed(M + N)
    K = 64
    a = torch.randn(M, K, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(N, K, device=DEV, dtype=torch.bfloat16)
    bias = (torch.randn(N + shift, device=DEV) * 8).to(dtype)[shift:]   # shift 1: not 16-byte aligned
    y = O.gemm(a, b, bias=bias, out_dtype=torch.float32, impl=impl)
    O.check_status()
    ref = a.double() @ b.double().t() + bias.double()
    # fp32 accumulation of 64 products of magnitude ~1 plus one rounding of the biased sum (|y| < 64)
    assert (y.double() - ref).abs().max().item() < 64 * 2.0 ** -22
