"""Attention backward at the edges of its 128-row tiles: ragged lengths, GQA rings longer than the tile ring, masks."""
import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Tq,Tk,Hq,Hkv,causal,window", [
    (1, 1, 1, 1, 1, True, 0), (2, 64, 64, 2, 2, True, 0), (1, 127, 127, 4, 2, True, 0), (1, 128, 128, 8, 1, True, 0),
    (2, 129, 129, 2, 1, True, 0), (1, 700, 700, 8, 2, True, 0), (1, 1500, 1500, 2, 2, False, 0), (1, 200, 513, 4, 1, True, 0),
    (1, 300, 130, 2, 2, True, 0), (1, 1000, 1000, 4, 2, True, 65), (1, 900, 900, 2, 1, True, 257), (1, 77, 640, 2, 2, False, 0),
    # streams long enough for 128-row tiles at head dimension 128, in one pass or both
    (2, 1301, 1301, 4, 2, True, 0), (1, 1900, 1900, 2, 1, True, 700), (1, 33, 1500, 4, 1, True, 0), (1, 1500, 40, 2, 2, False, 0)])
def test_gradients(D, B, Tq, Tk, Hq, Hkv, causal, window):
    torch.manual_seed(Tq + Tk)
    q = torch.randn(B, Tq, Hq, D, device=DEV).bfloat16().requires_grad_()
    k, v = (torch.randn(B, Tk, Hkv, D, device=DEV).bfloat16().requires_grad_() for _ in range(2))
    do = torch.randn(B, Tq, Hq, D, device=DEV).bfloat16()
    o = O.flash_attention(q, k, v, causal=causal, window=window)
    got = torch.autograd.grad(o, (q, k, v), do)
    O.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = torch.autograd.grad(O.attention_reference(qr, kr, vr, causal, window=window), (qr, kr, vr), do.float())
    for g, r in zip(got, ref):
        # P, dS, O and the results rounded to bf16; a query with a single key has a zero gradient for q and k
        assert torch.isfinite(g).all()
        assert (g.float() - r).norm().item() <= 1.2e-2 * r.norm().item() + 1e-2 * (Tk == 1)
        assert (g.float() - r).abs().max().item() <= 6e-2 * max(1.0, r.abs().max().item())


def test_packed_segments():
    torch.manual_seed(0)
    T, H, D = 777, 4, 128
    from tensorplay_b200.ops.attention import segment_bounds
    lo, hi = segment_bounds(torch.tensor([0, 5, 128, 400, 401, 777], device=DEV), T)
    lo, hi = lo.view(1, T), hi.view(1, T)
    q, k, v = (torch.randn(1, T, H, D, device=DEV).bfloat16().requires_grad_() for _ in range(3))
    do = torch.randn(1, T, H, D, device=DEV).bfloat16()
    got = torch.autograd.grad(O.flash_attention(q, k, v, True, seg_start=lo, seg_end=hi), (q, k, v), do)
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = torch.autograd.grad(O.attention_reference(qr, kr, vr, True, seg_start=lo, seg_end=hi), (qr, kr, vr), do.float())
    for g, r in zip(got, ref):
        assert ((g.float() - r).norm() / r.norm()).item() < 1.2e-2


@pytest.mark.parametrize("passes", ["both", "dq"])
@pytest.mark.parametrize("Tq,Tk,Hq,Hkv,causal,window,packed", [
    (129, 129, 8, 8, True, 0, False), (70, 70, 8, 2, True, 0, False), (300, 300, 4, 2, True, 100, False),
    (100, 200, 8, 4, True, 0, False), (200, 77, 4, 4, False, 0, False), (1, 65, 8, 2, True, 0, False),
    (260, 260, 8, 4, True, 0, True)])
def test_many_short_sequences(Tq, Tk, Hq, Hkv, causal, window, packed, passes):
    """Head dimension 64 with at least six CTAs per SM, in both passes or, with few key heads, in the dQ pass only: two
    CTAs share an SM and its TMEM."""
    from tensorplay_b200.ops.attention import segment_bounds
    need = 6 * torch.cuda.get_device_properties(0).multi_processor_count
    if passes == "dq":
        Hkv, Hq = 1, 16
    B = -(-need // (-(-Tk // 128) * Hkv)) if passes == "both" else -(-need // (-(-Tq // 128) * Hq))
    if passes == "both":
        B = max(B, -(-need // (-(-Tq // 128) * Hq)))
    assert B * -(-Tq // 128) * Hq >= need and (B * -(-Tk // 128) * Hkv >= need) == (passes == "both")
    torch.manual_seed(Tq + Tk)
    q, do = (torch.randn(B, Tq, Hq, 64, device=DEV).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Tk, Hkv, 64, device=DEV).bfloat16() for _ in range(2))
    kw = {}
    if packed:
        lo, hi = segment_bounds(torch.tensor([0, 5, 128, 131, Tq], device=DEV), Tq)
        kw = dict(seg_start=lo.repeat(B, 1), seg_end=hi.repeat(B, 1))
    for t in (q, k, v):
        t.requires_grad_()
    got = torch.autograd.grad(O.flash_attention(q, k, v, causal, window=window, **kw), (q, k, v), do)
    O.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = torch.autograd.grad(O.attention_reference(qr, kr, vr, causal, window=window, **kw), (qr, kr, vr), do.float())
    for g, r in zip(got, ref):   # bounds as above
        assert torch.isfinite(g).all()
        assert (g.float() - r).norm().item() <= 1.2e-2 * r.norm().item()
        assert (g.float() - r).abs().max().item() <= 6e-2 * max(1.0, r.abs().max().item())
