"""Cached passes of a decoder that one native call must leave to the pass layer by layer: what that one refuses stays refused, what
it calls is called, and its results are its own."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200 import _native
from tensorplay_b200.models.llama import Llama, LlamaBlock, LlamaConfig
from tensorplay_b200.nn.cache import DynamicCache, StaticCache

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _model(**kw):
    cfg = LlamaConfig.tiny(hidden_size=256, num_heads=4, num_kv_heads=2, head_dim=64, ffn_size=328, vocab_size=520, num_layers=2,
                           **kw)
    m = Llama(cfg, device=DEV, dtype=torch.bfloat16)
    m.reset_parameters(seed=0)
    return m


@pytest.fixture
def seen(monkeypatch):
    """The native calls of whole passes."""
    L, seen = _native.kernels(), []
    own = L.tpb_llama_cached
    monkeypatch.setattr(L, "tpb_llama_cached", lambda *a: seen.append(1) or own(*a), raising=False)
    return seen


@torch.no_grad()
def _pass(m, tok, cache):
    return m(tok, past_key_values=cache)


def test_short_tables_raise(monkeypatch, seen):
    """Rotary tables of the class's own that end before the last position."""
    m, cache = _model(), DynamicCache()
    tok = torch.randint(0, 520, (2, 9), device=DEV)
    tables = O.rope_tables(8, 64, device=DEV)
    monkeypatch.setattr(Llama, "rope_tables", lambda self, n, device: tables)
    _pass(m, tok[:, :8].contiguous(), cache)
    assert seen == [1]
    with pytest.raises(IndexError):
        _pass(m, tok[:, 8:].contiguous(), cache)
    assert seen == [1] and cache.get_seq_length(0) == 8


def test_buffers_that_did_not_grow_with_the_limit(seen):
    m, cache = _model(), StaticCache(8)
    tok = torch.randint(0, 520, (2, 9), device=DEV)
    _pass(m, tok[:, :8].contiguous(), cache)
    cache.max_seq_len = 64   # the buffers hold 8 tokens
    with pytest.raises(ValueError):
        _pass(m, tok[:, 8:].contiguous(), cache)
    assert seen == [1] and cache.get_seq_length(0) == 8


@pytest.mark.parametrize("name", ["_plain_inference", "_weights", "_shapes_as_configured", "_attend_cached", "_infer_cached"])
def test_replaced_on_the_block_class(monkeypatch, seen, name):
    """What the pass layer by layer asks of a block is asked where the class has another one."""
    m, own = _model(), []
    f = getattr(LlamaBlock, name)
    monkeypatch.setattr(LlamaBlock, name, lambda *a: own.append(1) or f(*a))
    if name == "_attend_cached":   # of a block that goes operator by operator
        monkeypatch.setattr(LlamaBlock, "_plain_inference", lambda *a: False)
    tok = torch.randint(0, 520, (2, 9), device=DEV)
    _pass(m, tok, DynamicCache())
    assert own == [1, 1] and not seen


def test_operators_of_a_block_that_says_it_is_not_plain(monkeypatch, seen):
    m, own = _model(), []
    monkeypatch.setattr(LlamaBlock, "_plain_inference", lambda *a: False)
    for name in ("apply_rope", "swiglu_packed"):
        f = getattr(O, name)
        monkeypatch.setattr(O, name, lambda *a, f=f, name=name: own.append(name) or f(*a))
    _pass(m, torch.randint(0, 520, (2, 9), device=DEV), DynamicCache())
    assert own == ["apply_rope", "swiglu_packed"] * 2 and not seen


def _both(m, call):
    """``call`` on the model as it is and with a hook that sends it layer by layer: two results or two refusals."""
    out = []
    for hook in (False, True):
        handle = m.layers[0].register_forward_hook(lambda *a: None) if hook else None
        try:
            out.append(call())
        except Exception as e:
            out.append((type(e), str(e)))
        if handle is not None:
            handle.remove()
    return out


def test_norm_weight_of_another_type(seen):
    m = _model()
    m.final_norm = torch.nn.Parameter(m.final_norm.detach().float())
    tok = torch.randint(0, 520, (2, 9), device=DEV)
    a, b = _both(m, lambda: _pass(m, tok, DynamicCache()))
    assert not seen and (torch.equal(a, b) if isinstance(a, torch.Tensor) else a == b)


def test_weight_of_other_strides(seen):
    m = _model()
    m.layers[1].wo = torch.nn.Parameter(m.layers[1].wo.detach().t().contiguous().t())
    tok = torch.randint(0, 520, (2, 9), device=DEV)
    a, b = _both(m, lambda: _pass(m, tok, DynamicCache()))
    assert not seen and torch.equal(a, b)


def test_with_gradients(seen):
    m = _model()
    tok = torch.randint(0, 520, (2, 8), device=DEV)

    def call():
        m.zero_grad(set_to_none=True)
        m(tok, past_key_values=DynamicCache()).float().square().sum().backward()
        return [p.grad for p in m.parameters()]

    a, b = _both(m, call)
    assert not seen and len(a) == 15 and all(torch.equal(x, y) and x.abs().sum() > 0 for x, y in zip(a, b))
