"""Attention where scores outgrow the running reference of the exponentials: in every column of a streamed tile, whether it is
handed over first (0..95) or last (96..127) and whether its exponentials are taken by the special-function unit or by the
polynomial, by less than the reference is allowed to lag, by more, and beyond the range of exp2 and of its exponent field."""
import math

import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200.ops.attention import flash_fwd

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(T, D, at, nats):
    torch.manual_seed(at + D)
    u = torch.randn(D, device=DEV)
    u /= u.norm()
    q = (torch.randn(1, T, 2, D, device=DEV) * 0.1 + u * math.sqrt(D)).bfloat16()
    k = torch.randn(1, T, 1, D, device=DEV) * 0.5
    k -= (k @ u).unsqueeze(-1) * u   # scores near zero, but for key `at`
    k[:, at] += u * nats
    return q, k.bfloat16(), torch.randn(1, T, 1, D, device=DEV).bfloat16()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("nats", [2.0, 5.0, 30.0, 400.0])
@pytest.mark.parametrize("at", [128, 223, 224, 255, 300, 383])
def test_growing_scores(D, causal, nats, at):
    T = 517
    q, k, v = _inputs(T, D, at, nats)
    o = O.flash_attention(q, k, v, causal=causal)
    O.check_status()
    ref = O.attention_reference(q.float(), k.float(), v.float(), causal)
    # P and O are rounded to bf16 (2^-9 each); both errors together, twice
    assert ((o.float() - ref).norm() / ref.norm()).item() < 8e-3
    assert (o.float() - ref).abs().max().item() < 8e-3 * ref.abs().max().item() * 2


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("nats", [2.0, 5.0, 30.0, 60.0, 88.0, 89.0, 90.0, 95.0, 100.0, 140.0, 150.0, 177.0, 178.0, 200.0, 250.0,
                                  260.0, 266.0, 300.0, 350.0, 360.0, 400.0])
def test_growth_in_every_column(D, causal, nats):
    """Sequence ``b`` has its outgrown score in column ``b`` of the second tile; the second head sees it negated. Output, LSE
    and gradients against fp32, each within what its roundings can add up to."""
    B, T, at = 128, 517, 128
    torch.manual_seed(D)
    u = torch.randn(D, device=DEV)
    u /= u.norm()
    sign = torch.tensor([1.0, -1.0], device=DEV).view(1, 1, 2, 1)
    q = (torch.randn(B, T, 2, D, device=DEV) * 0.1 + sign * u * math.sqrt(D)).bfloat16().requires_grad_()
    k = torch.randn(B, T, 1, D, device=DEV) * 0.5
    k -= (k @ u).unsqueeze(-1) * u   # scores near zero, but for the key of the column
    k[torch.arange(B), at + torch.arange(B), 0] += u * nats
    k = k.bfloat16().requires_grad_()
    v = torch.randn(B, T, 1, D, device=DEV).bfloat16().requires_grad_()
    do = torch.randn(B, T, 2, D, device=DEV).bfloat16()
    scale = 1.0 / math.sqrt(D)
    o = O.flash_attention(q, k, v, causal=causal)
    got = torch.autograd.grad(o, (q, k, v), do)
    _, lse = flash_fwd(q.detach(), k.detach(), v.detach(), causal, scale)
    O.check_status()

    with torch.no_grad():
        qf, dof = (t.float().transpose(1, 2) for t in (q, do))              # [B, 2, T, D]
        kf, vf = (t.float().transpose(1, 2).expand(B, 2, T, D) for t in (k, v))
        s = qf @ kf.transpose(2, 3) * scale
        if causal:
            s.masked_fill_(torch.ones(T, T, dtype=torch.bool, device=DEV).triu(1), float("-inf"))
        ref_lse = torch.logsumexp(s, -1)
        p = torch.exp(s - ref_lse.unsqueeze(-1))
        ref_o = p @ vf
        # scores: D products are added in fp32 on both sides, then scaled; exp2's cubic is 1e-4 off
        ds_err = 2 * D * 2.0 ** -24 * (nats + 8)
        assert ((lse[:, :, :T] - ref_lse).abs() <= ds_err + 2e-4).all()
        # P and O are rounded to bf16 (2^-9 each), P is exp of a score
        p_err = 2.0 ** -9 + 2e-4 + ds_err
        assert ((o.transpose(1, 2).float() - ref_o).abs() <= p_err * (p @ vf.abs()) + 2.0 ** -8 * ref_o.abs() + 1e-6).all()
        dp = dof @ vf.transpose(2, 3)
        delta = (dof * ref_o).sum(-1, keepdim=True)
        ds = p * (dp - delta)
        # dS: P once more, delta from the rounded O, dS itself rounded to bf16
        e = p * (dp - delta).abs() * (2 * p_err + 2.0 ** -8) + p * (dof * ref_o).abs().sum(-1, keepdim=True) * (p_err + 2.0 ** -8)
        dq, tol_q = ds @ kf * scale, e @ kf.abs() * scale
        dk, tol_k = (ds.transpose(2, 3) @ qf * scale).sum(1, keepdim=True), (e.transpose(2, 3) @ qf.abs() * scale).sum(1, keepdim=True)
        dv = (p.transpose(2, 3) @ dof).sum(1, keepdim=True)
        tol_v = p_err * (p.transpose(2, 3) @ dof.abs()).sum(1, keepdim=True)
        for g, ref, tol in zip(got, (dq, dk, dv), (tol_q, tol_k, tol_v)):
            assert ((g.transpose(1, 2).float() - ref).abs() <= 2 * tol + 2.0 ** -8 * ref.abs() + 1e-5).all()


def test_nan_and_infinity_stay_in_their_rows():
    q, k, v = _inputs(517, 128, 300, 5.0)
    q[0, 400, 0, 3] = float("nan")
    q[0, 130, 1, 5] = float("inf")
    o = O.flash_attention(q, k, v, causal=False)
    ref = O.attention_reference(q.float(), k.float(), v.float(), False)
    O.check_status()
    assert torch.isnan(o[0, 400, 0]).all() and torch.isnan(o[0, 130, 1]).all()
    rest = torch.ones(517, 2, dtype=torch.bool, device=DEV)
    rest[400, 0] = rest[130, 1] = False
    assert ((o[0][rest].float() - ref[0][rest]).norm() / ref[0][rest].norm()).item() < 8e-3
