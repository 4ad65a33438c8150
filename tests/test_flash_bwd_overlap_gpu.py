"""The two passes of the attention backward overlap: what follows in the stream, and a captured graph, sees both complete."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200.ops.attention import flash_bwd, flash_fwd

pytestmark = pytest.mark.gpu
DEV = "cuda"


# dKV passes that outlast their dQ pass (many query heads per key head, few queries), the other way round, and both forms
@pytest.mark.parametrize("B,Tq,Tk,Hq,Hkv,D", [(1, 1100, 1100, 16, 1, 128), (1, 64, 3000, 8, 8, 128), (2, 300, 300, 8, 2, 64),
                                              (1, 2000, 2000, 8, 1, 64), (16, 200, 200, 64, 64, 64)])
def test_followers_and_graphs_see_both_passes(B, Tq, Tk, Hq, Hkv, D):
    torch.manual_seed(Tk)
    q, do = (torch.randn(B, Tq, Hq, D, device=DEV).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Tk, Hkv, D, device=DEV).bfloat16() for _ in range(2))
    o, lse = flash_fwd(q, k, v, True, D ** -0.5)
    want = [t.clone() for t in flash_bwd(do, q, k, v, o, lse, True, D ** -0.5)]
    torch.cuda.synchronize()
    out = [torch.empty_like(t) for t in (q, k, v)]

    def passes():
        for t in out:
            t.fill_(float("nan"))
        flash_bwd(do, q, k, v, o, lse, True, D ** -0.5, dq=out[0], dk=out[1], dv=out[2])
        return [t.clone() for t in out]

    for _ in range(4):
        for a, b in zip(passes(), want):   # neither pass has atomics: the same bits every time
            assert torch.equal(a, b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = passes()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    O.check_status()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
