"""Cross-entropy forward around the sizes at which its blocks change: rows by SMs, logits by the rounds of a block."""
import pytest
import torch

import tensorplay_b200.ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("V", [16384, 16385, 16392, 40960, 40965, 50257, 128256])
@pytest.mark.parametrize("per_sm,more", [(0, 2), (1, 0), (1, 1), (2, 0), (2, 1)])
def test_forward(V, per_sm, more):
    rows = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    torch.manual_seed(V + rows)
    ld = (V + 7) // 8 * 8
    lg = (torch.randn(rows, ld, device=DEV) * 4).bfloat16()[:, :V]
    lg[0, : V // 2] = float("-inf")
    tgt = torch.randint(0, V, (rows,), device=DEV)
    tgt[0] = V - 1
    got = O.cross_entropy(lg, tgt, reduction="none")
    ref = torch.nn.functional.cross_entropy(lg.double(), tgt, reduction="none")
    # fp32 sum of at most V exponentials and one logarithm; logits below 2^5
    assert (got.double() - ref).abs().max().item() < 2e-5
