"""Routing and row exchange of the experts: more choices than one look-up holds, ragged widths, more experts than a warp."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200.parallel.moe import MoEWorkspace, expert_ffn_reference, expert_parallel_ffn, topk_route

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("T,H,E,k", [(3, 72, 40, 1), (60, 2120, 2, 2), (60, 64, 40, 9)])
def test_rows(T, H, E, k):
    torch.manual_seed(T)
    I = 64
    ws = MoEWorkspace(T, k, H, E, wait_s=5.0)
    x = torch.randn(T, H, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    idx, w, _ = topk_route(torch.randn(T, E, device=DEV), k)
    w = w.to(torch.bfloat16).requires_grad_()
    gu = (torch.randn(E, 2 * I, H, device=DEV, dtype=torch.bfloat16) * 0.05).requires_grad_()
    down = (torch.randn(E, H, I, device=DEV, dtype=torch.bfloat16) * 0.05).requires_grad_()
    y = expert_parallel_ffn(x, idx, w, gu, down, ws)
    g = torch.randn_like(y)
    got = [y] + list(torch.autograd.grad(y, (x, w, gu, down), g))
    O.check_status()
    leaves = [t.detach().float().requires_grad_() for t in (x, w, gu, down)]
    ref = expert_ffn_reference(leaves[0], idx, *leaves[1:])
    want = [ref] + list(torch.autograd.grad(ref, leaves, g.float()))
    for a, b in zip(got, want):
        # some four roundings to bf16 (2^-9 relative at most) lie between the leaves and each result, by norm
        assert ((a.float() - b).norm() / b.norm()).item() < 4 * 2.0 ** -9
