"""Attention forward where scores outgrow the running reference of the exponentials: in the keys of a tile that are handed
over first (0..95) or last (96..127), by less than the reference is allowed to lag, by more, and beyond the range of exp2."""
import math

import pytest
import torch

import tensorplay_b200.ops as O

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
