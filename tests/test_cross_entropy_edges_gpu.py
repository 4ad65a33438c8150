"""Cross-entropy forward: vocabulary sizes around a thread's vectors, rows that start with or hold masked logits."""
import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("V", [8, 13, 4096, 4104, 16384, 16397, 50304])
@pytest.mark.parametrize("masked", [0.0, 0.4])
def test_forward(V, masked):
    torch.manual_seed(V)
    ld = (V + 7) // 8 * 8
    lg = (torch.randn(9, ld, device=DEV) * 4).bfloat16()[:, :V]
    if masked:
        lg[:, : int(V * masked)] = float("-inf")     # whole vectors, from the first one on
        lg[3, :] = lg[3, :].clamp_min(torch.finfo(torch.bfloat16).min)
    tgt = torch.full((9,), V - 1, device=DEV)
    tgt[1] = -100
    got = O.cross_entropy(lg, tgt, reduction="none")
    ref = torch.nn.functional.cross_entropy(lg.double(), tgt, reduction="none")
    # fp32 sum of at most V exponentials and one logarithm; logits below 2^5
    assert (got.double() - ref).abs().max().item() < 2e-5
