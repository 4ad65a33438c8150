"""Cached passes of a decoder that one native call must leave to the pass layer by layer: what that one refuses stays refused, what
it calls is called, and its results are its own."""
import pytest
import torch

import tensorplay_b200.ops as O
from tensorplay_b200 import _native
from tensorplay_b200.models.llama import Llama, LlamaConfig
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
