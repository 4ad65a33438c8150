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


@pytest.mark.parametrize("M,N", [(256, 256), (130, 264), (513, 64), (129, 40), (300, 328)])
@pytest.mark.parametrize("pad,shift", [(0, 0), (8, 8), (8, 4), (3, 0)])
def test_bf16_stores(M, N, pad, shift):
    """Rows that leave as whole lines and those that cannot (last columns, unaligned output), and nothing beside them."""
    torch.manual_seed(M + N)
    a = torch.randn(M, 192, device=DEV, dtype=torch.bfloat16)
    b = torch.randn(N, 192, device=DEV, dtype=torch.bfloat16)
    bias = torch.randn(N, device=DEV, dtype=torch.bfloat16)
    ref = (a.double() @ b.double().t() + bias.double())
    buf = torch.full((M + 2, N + pad + shift), 7.0, device=DEV, dtype=torch.bfloat16)
    out = buf[:M, shift:shift + N]
    O.gemm(a, b, bias=bias, out=out, impl="pair")
    O.check_status()
    assert ((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 192 * 2.0 ** -20).all()
    rest = buf.clone()
    rest[:M, shift:shift + N] = 7.0
    assert (rest == 7.0).all()


@pytest.mark.parametrize("rows,N", [(1, 8), (7, 264), (33, 768), (4096, 40), (16384, 2304)])
def test_bias_gradient(rows, N):
    torch.manual_seed(rows)
    x = torch.randn(rows, 64, device=DEV, dtype=torch.bfloat16)
    w = torch.randn(N, 64, device=DEV, dtype=torch.bfloat16)
    b = torch.zeros(N, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(rows, N, device=DEV, dtype=torch.bfloat16)
    (db,) = torch.autograd.grad(O.linear(x, w, b), b, dy)
    ref = dy.double().sum(0)
    # fp32 sums of `rows` unit-variance terms (error a few ulp of a partial sum of size sqrt(rows)), rounded once to bf16
    tol = ref.abs() * 2.0 ** -8 + 64 * 2.0 ** -24 * rows ** 0.5 + 1e-6
    assert ((db.double() - ref).abs() <= tol).all()


@pytest.mark.parametrize("rows,H", [(1, 8), (5, 136), (600, 768), (3000, 1024)])
def test_norm_weight_gradients(rows, H):
    torch.manual_seed(H)
    x = torch.randn(rows, H, device=DEV, dtype=torch.bfloat16)
    w, b = (torch.randn(H, device=DEV, dtype=torch.bfloat16, requires_grad=True) for _ in range(2))
    dy = torch.randn(rows, H, device=DEV, dtype=torch.bfloat16)
    dw, db = torch.autograd.grad(O.layer_norm(x, w, b), (w, b), dy)
    (dr,) = torch.autograd.grad(O.rms_norm(x, w), w, dy)
    xd, wd, bd = x.double(), w.detach().double().requires_grad_(), b.detach().double().requires_grad_()
    rw, rb = torch.autograd.grad(torch.nn.functional.layer_norm(xd, (H,), wd, bd, 1e-5), (wd, bd), dy.double())
    (rr,) = torch.autograd.grad(xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-5) * wd, wd, dy.double())
    for got, ref in ((dw, rw), (db, rb), (dr, rr)):
        tol = ref.abs() * 2.0 ** -8 + 1e-5 * rows ** 0.5
        assert ((got.double() - ref).abs() <= tol).all()
