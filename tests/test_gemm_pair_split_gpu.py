"""Products with fewer tiles than CTA pairs: the reduction shared by the pairs of a cluster, at the edges of tiles and splits."""
import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _check(M, N, K, a_mn, b_mn, out_dtype=torch.bfloat16, bias=None, accumulate=False, alpha=1.0):
    torch.manual_seed(M * 7 + N * 3 + K)
    a = torch.randn((K, M + (-M) % 8) if a_mn else (M, K), device=DEV).bfloat16()
    b = torch.randn((K, N + (-N) % 8) if b_mn else (N, K), device=DEV).bfloat16()
    a, b = (a[:, :M] if a_mn else a), (b[:, :N] if b_mn else b)
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


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [(768, 768, 16384), (2304, 768, 4096), (136, 264, 4104), (1031, 520, 2472), (256, 72, 65536)])
def test_small_output_long_reduction(M, N, K, a_mn, b_mn):
    _check(M, N, K, a_mn, b_mn)


@pytest.mark.parametrize("kw", [dict(out_dtype=torch.float32, bias=torch.float32, accumulate=True, alpha=0.5),
                                dict(bias=torch.bfloat16, accumulate=True), dict(out_dtype=torch.float32)])
def test_epilogue(kw):
    _check(500, 1036, 8192, False, False, **kw)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("M,N,K", [(1000, 4096, 2048), (2500, 1032, 4096), (200, 14336, 512), (1024, 1024, 64)])
def test_less_than_a_wave_of_pairs(M, N, K, a_mn, b_mn):
    """Products that stay whole: on CTA pairs, or on single CTAs."""
    _check(M, N, K, a_mn, b_mn)
