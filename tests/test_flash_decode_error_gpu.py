"""Attention of at most eight query rows to a KV head: as near to 64 bits as the rounding of its result."""
import math

import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


# rows to a KV head: 1, 4, 8 (of one token or several); one split, a cluster of them, two launches; short and ragged keys
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Tq,Tk,Hq,Hkv,window", [(8, 1, 16381, 32, 8, 0), (2, 1, 9000, 8, 8, 0), (1, 1, 30000, 8, 2, 0),
                                                   (3, 2, 777, 8, 2, 0), (1, 8, 4100, 4, 4, 0), (4, 1, 50, 16, 2, 0),
                                                   (5, 1, 17, 8, 1, 0), (2, 4, 3000, 8, 4, 500)])
def test_error_is_the_rounding_of_the_result(D, B, Tq, Tk, Hq, Hkv, window):
    torch.manual_seed(Tk + D)
    q = torch.randn(B, Tq, Hq, D, device=DEV).bfloat16()
    k, v = (torch.randn(B, Tk, Hkv, D, device=DEV).bfloat16() for _ in range(2))
    with torch.no_grad():
        o = O.flash_attention(q, k, v, causal=True, window=window)
    qd, kd, vd = (t.double().transpose(1, 2) for t in (q, k, v))
    kd, vd = (t.repeat_interleave(Hq // Hkv, 1) for t in (kd, vd))
    s = qd @ kd.transpose(2, 3) / math.sqrt(D)
    at, key = torch.arange(Tq, device=DEV).view(-1, 1) + (Tk - Tq), torch.arange(Tk, device=DEV).view(1, -1)
    hide = key > at
    if window:
        hide |= key < at - window + 1
    ref = (torch.softmax(s.masked_fill(hide, float("-inf")), -1) @ vd).transpose(1, 2)
    err, own = ((t.double() - ref).norm() / ref.norm() for t in (o, ref.bfloat16()))
    # besides: scores and sums in fp32, exponentials to 2^-22, probabilities to 2^-17, some 2e-5 of a result of 1.7e-3; one per
    # cent of the own error leaves room for 2.3e-4. Probabilities in one bf16 number make it 1.2 times as large and more.
    assert err <= 1.01 * own
