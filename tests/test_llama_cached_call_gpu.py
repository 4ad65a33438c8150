"""A cached pass of a whole decoder as one native call: the bits of the pass layer by layer, and what keeps it from being taken."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200 import _native
from tensorplay_b200.models.llama import Llama, LlamaConfig
from tensorplay_b200.nn.cache import DynamicCache, StaticCache

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _model(D=64, **kw):
    cfg = LlamaConfig.tiny(hidden_size=256, num_heads=4, num_kv_heads=2, head_dim=D, ffn_size=328, vocab_size=520,
                           num_layers=2, **kw)
    m = Llama(cfg, device=DEV, dtype=torch.bfloat16)
    m.reset_parameters(seed=0)
    return m


def _calls(monkeypatch):
    """Counts the native calls of whole passes."""
    L, seen = _native.kernels(), []
    own = L.tpb_llama_cached
    monkeypatch.setattr(L, "tpb_llama_cached", lambda *a: seen.append(1) or own(*a), raising=False)
    return seen


def _run(m, tok, cuts, cache, pos=False):
    out, a = [], 0
    with torch.no_grad():
        for b in cuts:
            p = torch.arange(a, b, device=DEV).expand(tok.shape[0], -1) if pos else None
            out.append(m(tok[:, a:b], position_ids=p, past_key_values=cache))
            a = b
    return out


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,cuts", [(1, (1, 2, 37, 38)), (3, (42, 43, 60)), (128, (1, 2)), (4, (32, 33)), (1, (128, 129, 150)),
                                    (2, (65, 66))])   # the last: a prompt of more than 128 rows goes layer by layer
@pytest.mark.parametrize("tie", [False, True])
@pytest.mark.parametrize("make,pos", [(DynamicCache, False), (lambda: StaticCache(160), True)])
def test_same_bits_as_layer_by_layer(monkeypatch, D, B, cuts, tie, make, pos):
    m = _model(D, tie_embeddings=tie, max_seq_len=256)
    tok = torch.randint(0, 520, (B, cuts[-1]), device=DEV)
    seen = _calls(monkeypatch)
    fast_cache, slow_cache = make(), make()
    fast = _run(m, tok, cuts, fast_cache, pos)
    assert len(seen) == sum(B * (b - a) <= 128 for a, b in zip((0,) + cuts, cuts))
    m.layers[0].register_forward_hook(lambda *a: None)
    n = len(seen)
    slow = _run(m, tok, cuts, slow_cache, pos)
    assert len(seen) == n
    O.check_status()
    for f, s in zip(fast, slow):
        assert torch.equal(f, s)
    for i in range(2):
        assert fast_cache.get_seq_length(i) == slow_cache.get_seq_length(i) == cuts[-1]
        assert torch.equal(fast_cache._k[i][:, :, :cuts[-1]], slow_cache._k[i][:, :, :cuts[-1]])


def test_long_cache(monkeypatch):
    """Keys split with partial rows in memory."""
    m = _model(128, max_seq_len=9000)
    seen = _calls(monkeypatch)
    tok = torch.randint(0, 520, (1, 8201), device=DEV)
    outs = []
    for hook in (False, True):
        if hook:
            m.layers[1].register_forward_pre_hook(lambda *a: None)
        outs.append(_run(m, tok, (8200, 8201), DynamicCache())[1])
    assert len(seen) == 1 and torch.equal(outs[0], outs[1])
    O.check_status()


@pytest.mark.parametrize("how", ["hook", "subclass", "method", "cache_method", "cache_class", "float", "transposed", "class_method",
                                 "grad", "global_hook"])
def test_goes_layer_by_layer(monkeypatch, how):
    m, cache = _model(), DynamicCache()
    tok = torch.randint(0, 520, (2, 9), device=DEV)
    seen, own = _calls(monkeypatch), []
    if how == "hook":
        m.layers[1].register_forward_pre_hook(lambda *a: own.append(1))
    elif how == "subclass":
        class Mine(Llama):
            def head(self, x, targets=None):
                own.append(1)
                return super().head(x, targets)
        m.__class__ = Mine
    elif how == "method":
        f = m.head
        m.head = lambda *a: own.append(1) or f(*a)
    elif how == "cache_method":
        f = cache.update
        cache.update = lambda *a: own.append(1) or f(*a)
    elif how == "cache_class":
        class Mine(DynamicCache):
            def update(self, *a):
                own.append(1)
                return super().update(*a)
        cache = Mine()
    elif how == "float":
        m.final_norm = torch.nn.Parameter(m.final_norm.detach().float())
        own.append(1)
    elif how == "transposed":
        w = m.layers[1].wo
        m.layers[1].wo = torch.nn.Parameter(w.detach().t().contiguous().t())
        own.append(1)
    elif how == "class_method":
        f = Llama.embed_tokens
        monkeypatch.setattr(Llama, "embed_tokens", lambda self, t: own.append(1) or f(self, t))
    elif how == "global_hook":
        handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: own.append(1))
    if how == "grad":
        m(tok[:, :8].contiguous(), past_key_values=cache).sum().backward()   # weight gradients take rows in eights
        own.append(1)
    elif how == "float":
        with pytest.raises(Exception):   # as before: the norm refuses another dtype, or a product does
            with torch.no_grad():
                m(tok, past_key_values=cache)
                raise TypeError
    else:
        with torch.no_grad():
            m(tok, past_key_values=cache)
    if how == "global_hook":
        handle.remove()
    assert own and not seen


def test_full_static_cache_raises():
    m, cache = _model(), StaticCache(8)
    tok = torch.randint(0, 520, (2, 9), device=DEV)
    with torch.no_grad():
        m(tok[:, :8].contiguous(), past_key_values=cache)
        with pytest.raises(ValueError):
            m(tok[:, 8:].contiguous(), past_key_values=cache)
    assert cache.get_seq_length(0) == 8


@pytest.mark.parametrize("B", [1, 5, 40])
def test_chained_launches_repeat(B):
    """Kernels of the call start before the ones they depend on have ended: many steps, back to back, bit by bit."""
    m = _model(64, max_seq_len=256)
    tok = torch.randint(0, 520, (B, 70), device=DEV)
    cuts = tuple(range(3, 71))
    fast = [_run(m, tok, cuts, DynamicCache()) for _ in range(3)]
    m.layers[0].register_forward_hook(lambda *a: None)
    slow = _run(m, tok, cuts, DynamicCache())
    O.check_status()
    for run in fast:
        for f, s in zip(run, slow):
            assert torch.equal(f, s)


def test_capture():
    m, cache = _model(128, max_seq_len=256), StaticCache(64)
    tok = torch.randint(0, 520, (3, 21), device=DEV)
    want = _run(m, tok, (20, 21), cache)[1].clone()
    with torch.no_grad():
        for i in range(2):
            cache._len[i] = 20
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = m(tok[:, 20:], past_key_values=cache)
        for _ in range(3):
            got.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(got, want)
    O.check_status()
