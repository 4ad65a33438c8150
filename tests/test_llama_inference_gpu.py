"""The native halves of the decoder block against the operators one by one, and what keeps them from being used."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200.models.llama import Llama, LlamaConfig
from tensorplay_b200.nn.cache import DynamicCache, PagedCache, SlidingWindowCache, StaticCache
from tensorplay_b200.utils.flop_counter import FlopCounterMode

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _model(D=64, **kw):
    cfg = LlamaConfig.tiny(hidden_size=256, num_heads=4, num_kv_heads=2, head_dim=D, ffn_size=328, vocab_size=512,
                           num_layers=2, **kw)
    m = Llama(cfg, device=DEV, dtype=torch.bfloat16)
    m.reset_parameters(seed=0)
    return m


def _run(m, tok, cuts, cache, grad, pos=False):
    out, a = [], 0
    for b in cuts:
        p = torch.arange(a, b, device=DEV).expand(tok.shape[0], -1) if pos else None
        with torch.set_grad_enabled(grad):
            out.append(m(tok[:, a:b], position_ids=p, past_key_values=cache).detach())
        a = b
    return torch.cat(out, 1)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,cuts", [(1, (7, 8, 9, 30)), (3, (1, 2, 60, 61)), (5, (50, 51)), (2, (300, 301, 317))])
@pytest.mark.parametrize("pos", [False, True])
def test_matches_single_operators(D, B, cuts, pos):
    m = _model(D, max_seq_len=512)
    tok = torch.randint(0, 512, (B, cuts[-1]), device=DEV)
    calls = []
    for layer in m.layers:
        layer.register_forward_hook(lambda *a: calls.append(1))
    fast = _run(m, tok, cuts, DynamicCache(), False, pos)
    assert len(calls) == 2 * len(cuts)
    slow = _run(m, tok, cuts, DynamicCache(), True, pos)   # gradients on: operator by operator
    O.check_status()
    # the same kernels but for one rounding of the residual sum per layer
    assert ((fast.float() - slow.float()).norm() / slow.float().norm()).item() < 1e-2


@pytest.mark.parametrize("make", [lambda: StaticCache(64), lambda: PagedCache(16), lambda: SlidingWindowCache(64)])
def test_cache_kinds(make):
    m = _model()
    tok = torch.randint(0, 512, (2, 40), device=DEV)
    with torch.no_grad():
        fast = _run(m, tok, (33, 34, 40), make(), False)
        blocks = [type(b)._plain_inference for b in m.layers]
        for b in m.layers:
            b._plain_inference = lambda *a: False
        slow = _run(m, tok, (33, 34, 40), make(), False)
    assert blocks and ((fast.float() - slow.float()).norm() / slow.float().norm()).item() < 1e-2


def test_falls_back_for_observers_and_other_tensors():
    m = _model()
    x = torch.randn(1, 4, 256, device=DEV).bfloat16()
    cos, sin = m.rope_tables(16, x.device)
    blk = m.layers[0]
    with torch.no_grad():
        assert blk._plain_inference(x, cos, sin)
        assert not blk._plain_inference(x.float(), cos, sin)
        assert not blk._plain_inference(x.transpose(0, 1).expand(4, 3, 256), cos, sin)
        with FlopCounterMode(display=False):
            assert not blk._plain_inference(x, cos, sin)
        with torch.autograd.forward_ad.dual_level():
            assert not blk._plain_inference(x, cos, sin)
        blk.wo = torch.nn.Parameter(blk.wo.detach().t().contiguous().t())
        assert not blk._plain_inference(x, cos, sin)
    assert not m.layers[1]._plain_inference(x, cos, sin)   # gradients on


def test_pair_append_strides():
    B, H, T, D = 2, 3, 5, 64
    cache = torch.zeros(2, B, H, 20, D, device=DEV, dtype=torch.bfloat16)
    src = torch.randn(B, T, 2 * H, D, device=DEV).bfloat16()
    k, v = src[:, :, :H].transpose(1, 2), src[:, :, H:].transpose(1, 2)
    from tensorplay_b200.ops.decode import kv_append_pair
    kv_append_pair(cache[0], cache[1], k, v, 9)
    assert torch.equal(cache[0][:, :, 9:14], k) and torch.equal(cache[1][:, :, 9:14], v)
    assert cache[:, :, :, :9].abs().max() == 0 and cache[:, :, :, 14:].abs().max() == 0


@pytest.mark.parametrize("ffn", [264, 392])
def test_pruned_and_widened_ffn(ffn):
    """A block whose FFN was replaced by one of another width than configured."""
    m = _model()
    with torch.no_grad():
        for blk in m.layers:
            blk.w_gate_up = torch.nn.Parameter(torch.randn(2 * ffn, 256, device=DEV).mul(0.02).bfloat16())
            blk.w_down = torch.nn.Parameter(torch.randn(256, ffn, device=DEV).mul(0.02).bfloat16())
    tok = torch.randint(0, 512, (2, 30), device=DEV)
    fast = _run(m, tok, (29, 30), DynamicCache(), False)
    slow = _run(m, tok, (29, 30), DynamicCache(), True)
    O.check_status()
    assert torch.equal(fast, slow)   # the same operators


def test_wrong_sizes_raise():
    m = _model()
    blk, (cos, sin) = m.layers[0], m.rope_tables(16, torch.device(DEV))
    with torch.no_grad():
        with pytest.raises(ValueError):
            blk(torch.zeros(1, 4, 264, device=DEV, dtype=torch.bfloat16), cos, sin, None, DynamicCache())
        for pos in (torch.arange(4, device=DEV).view(1, 4), torch.arange(8).view(2, 4)):   # one row for two, and on the host
            with pytest.raises(ValueError):
                blk(torch.zeros(2, 4, 256, device=DEV, dtype=torch.bfloat16), cos, sin, pos, DynamicCache())
        blk.attn_norm.data = torch.empty(0, device=DEV, dtype=torch.bfloat16)   # as a sharding engine leaves it
        with pytest.raises(ValueError):
            blk(torch.zeros(1, 4, 256, device=DEV, dtype=torch.bfloat16), cos, sin, None, DynamicCache())


def test_own_cached_attention_is_called():
    m = _model()
    calls = []
    blk = m.layers[1]
    own = blk._attend_cached
    blk._attend_cached = lambda *a: calls.append(1) or own(*a)
    tok = torch.randint(0, 512, (2, 9), device=DEV)
    _run(m, tok, (8, 9), DynamicCache(), False)
    assert len(calls) == 2
