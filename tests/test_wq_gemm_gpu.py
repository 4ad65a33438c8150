"""Products with packed weights that are converted on their way to the tensor cores, against fp64 over the weights that
``dequantize_weight`` gives."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200 import _native
from tensorplay_b200.ops._common import status_word, stream_ptr
from tensorplay_b200.ops.quant import dequantize_weight, quantize_weight_int4, quantize_weight_int8, weight_only_linear

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _weights(N, K, bits, group, zero, g):
    w = torch.randn(N, K, generator=g, device=DEV) * 0.02
    if bits == 8:
        q, s = quantize_weight_int8(w, group)
        return q, s, None
    q, s, z = quantize_weight_int4(w, group)
    if zero == "none":
        z = None
    elif zero == "fraction":   # not what the quantiser makes: converted in fp32
        z = (z.float() + 0.3).bfloat16()
    elif zero == "mixed":      # rows of both kinds in one warp
        z = torch.where(torch.arange(N, device=DEV).view(-1, 1) % 7 == 0, z.float() - 0.5, z.float()).bfloat16()
    return q, s, z


def _check(y, x, w, bias):
    ref = x.double() @ w.double().t() + (bias.double() if bias is not None else 0.0)
    # products of bf16 values are exact in fp32; K of them are added with an error below K 2^-24 of the sum of their
    # magnitudes, and the result is rounded to bf16
    mag = x.double().abs() @ w.double().abs().t()
    assert ((y.double() - ref).abs() <= mag * x.shape[1] * 2.0 ** -24 + ref.abs() * 2.0 ** -8 + 1e-30).all()


# rows of x: one tile of 16, an odd one, more than one tile, more tiles than SMs; K of one, an odd number of blocks and more
# than the rings hold; N with a ragged last tile
@pytest.mark.parametrize("M", [1, 17, 129, 200, 577])
@pytest.mark.parametrize("N,K", [(8, 128), (136, 384), (1000, 1152), (4104, 2176)])
@pytest.mark.parametrize("bits,groups,zero,bias", [(4, 1, "whole", False), (4, 1, "none", True), (4, 1, "fraction", True),
                                                   (4, 1, "mixed", False), (4, 2, "whole", True), (8, 0, None, True),
                                                   (8, 1, None, False)])
def test_against_converted_weights(M, N, K, bits, groups, zero, bias):
    if groups == 2 and K % 256:
        K += 128
    g = torch.Generator(device=DEV)
    g.manual_seed(M + N + K)
    q, s, z = _weights(N, K, bits, 128 * groups, zero, g)
    x = (torch.randn(M, K + 24, generator=g, device=DEV) + 0.5).bfloat16()[:, :K]   # rows with a stride
    b = torch.randn(N, generator=g, device=DEV).bfloat16() if bias else None
    y = torch.full((M, N + 6), float("nan"), device=DEV, dtype=torch.bfloat16)
    code = _native.kernels().tpb_wq_gemm(
        x.data_ptr(), q.data_ptr(), s.data_ptr(), None if z is None else z.data_ptr(), None if b is None else b.data_ptr(),
        y.data_ptr(), M, N, K, bits, 128 * groups, x.stride(0), y.stride(0), status_word(x.device).data_ptr(), stream_ptr())
    O.check_status()
    assert code == 0 and torch.isnan(y[:, N:]).all()
    _check(y[:, :N], x, dequantize_weight(q, s, z, bits, 128 * groups), b)


def test_what_it_does_not_take():
    L = _native.kernels()
    x = torch.zeros(32, 256, device=DEV, dtype=torch.bfloat16)
    args = (x.data_ptr(), x.data_ptr(), x.data_ptr(), None, None, x.data_ptr())
    for M, N, K, bits, group in ((32, 16, 192, 8, 0), (32, 12, 256, 8, 0), (32, 16, 256, 4, 64), (32, 16, 768, 4, 384)):
        assert L.tpb_wq_gemm(*args, M, N, K, bits, group, 256, 16, status_word(x.device).data_ptr(), stream_ptr()) == -3
        assert not L.tpb_wq_gemm_pays(M, N, K, bits, group)
    assert not L.tpb_wq_gemm_pays(16, 28672, 8192, 4, 128)   # the GEMV does not round the weights


def test_linear_takes_it_without_gradients(monkeypatch):
    L, seen = _native.kernels(), []
    own = L.tpb_wq_gemm
    monkeypatch.setattr(L, "tpb_wq_gemm", lambda *a: seen.append(1) or own(*a), raising=False)
    g = torch.Generator(device=DEV)
    g.manual_seed(1)
    q, s, z = _weights(8192, 1024, 4, 128, "whole", g)
    w = dequantize_weight(q, s, z, 4, 128)
    x = torch.randn(3, 25, 1024, generator=g, device=DEV).bfloat16()
    y = weight_only_linear(x, q, s, z, None, 4, 128)
    assert seen == [1] and y.shape == (3, 25, 8192)
    _check(y.view(75, -1), x.view(75, -1), w, None)
    _check(weight_only_linear(x[:2, :24].transpose(0, 1), q, s, z, None, 4, 128).reshape(48, -1),
           x[:2, :24].transpose(0, 1).reshape(48, -1), w, None)
    n = len(seen)
    xg = x[:, :24].clone().requires_grad_()
    (gx,) = torch.autograd.grad(weight_only_linear(xg, q, s, z, None, 4, 128).float().sum(), xg)
    assert len(seen) == n and torch.isfinite(gx).all() and gx.abs().sum() > 0
