"""Products with few rows: every tile width of the kernel, edges of its tiles and of its reduction split."""
import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _check(M, N, K, a_mn, b_mn, out_dtype=torch.bfloat16, bias=None, accumulate=False, alpha=1.0, pad=0):
    torch.manual_seed(M * 7 + N * 3 + K)
    a = torch.randn((K, M + (-M) % 8 + pad) if a_mn else (M, K + pad), device=DEV).bfloat16()
    b = torch.randn((K, N + (-N) % 8 + pad) if b_mn else (N, K + pad), device=DEV).bfloat16()
    a, b = (a[:, :M] if a_mn else a[:, :K]), (b[:, :N] if b_mn else b[:, :K])
    out = torch.randn(M, N, device=DEV).to(out_dtype)
    ref = alpha * ((a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double())
    if bias is not None:
        bias = torch.randn(N, device=DEV).to(bias)
        ref = ref + bias.double()
    if accumulate:
        ref = ref + out.double()
    O.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=out, bias=bias, accumulate=accumulate, alpha=alpha)
    O.check_status()
    # one rounding to the output, and the fp32 accumulator: K / 16 steps that each cut at most an ulp (2^-23) of a
    # partial sum of K unit-variance products (below 2 sqrt(K) but for outliers)
    tol = 2.0 ** -8 * ref.abs() * (out_dtype == torch.bfloat16) + (K / 16 + 1) * 2.0 ** -23 * 2 * K ** 0.5 + 1e-6
    assert ((out.double() - ref).abs() <= tol).all()


@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("N,K", [(8, 8), (136, 72), (1000, 512), (4096, 4104)])
def test_few_rows(M, N, K, b_mn):
    _check(M, N, K, False, b_mn, pad=8)


@pytest.mark.parametrize("kw", [dict(out_dtype=torch.float32, bias=torch.float32, accumulate=True, alpha=0.5),
                                dict(bias=torch.bfloat16, accumulate=True), dict(bias=torch.float32)])
@pytest.mark.parametrize("M,N,K", [(5, 264, 2048), (100, 1036, 1024)])
def test_few_rows_epilogue(M, N, K, kw):
    _check(M, N, K, False, False, **kw)


@pytest.mark.parametrize("M,N,K", [(16, 40000, 72), (1, 40000, 4096), (17, 37888, 136), (32, 37896, 136), (33, 9472, 192),
                                   (64, 9480, 192), (65, 6272, 4096), (128, 4736, 64), (128, 4744, 64), (128, 6280, 4096),
                                   (16, 40000, 2040), (16, 40000, 2048), (32, 40000, 3072), (64, 11264, 3072), (65, 11272, 3072),
                                   (128, 11264, 3064), (128, 6272, 1024), (65, 6280, 1024), (128, 2688, 64), (100, 2696, 1016)])
def test_both_sides_of_the_choice(M, N, K):
    """Sizes on which the kernels of few and of more rows meet."""
    _check(M, N, K, False, M % 2 == 0)


def test_choice_by_the_kind_of_result():
    _check(40, 18944, 200, False, False, out_dtype=torch.float32, bias=torch.bfloat16)
    _check(64, 18816, 200, False, False, out_dtype=torch.float32, bias=torch.bfloat16)
    _check(64, 37888, 72, False, False, accumulate=True)
    _check(32, 40000, 72, False, False, accumulate=True)
    _check(16, 40000, 72, False, False, out_dtype=torch.float32, bias=torch.bfloat16)
