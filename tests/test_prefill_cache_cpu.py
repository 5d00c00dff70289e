"""What GemmaForCausalLM.prefill refuses before it launches anything (no device needed: the library is a stub that counts calls)."""
import pytest
import torch

from paligemma_multimodal_system_b200 import _lib, modeling_gemma
from paligemma_multimodal_system_b200.random_init import TINY_CONFIG


class _Library:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *a: self.calls.append(name) or 0


@pytest.mark.parametrize("layers,accepted", [(1, False), (2, True), (3, True)])
def test_a_cache_of_fewer_layers_is_refused(monkeypatch, layers, accepted):
    library = _Library()
    monkeypatch.setattr(_lib, "lib", lambda: library)
    monkeypatch.setattr(_lib, "stream", lambda: 0)
    c = TINY_CONFIG["text_config"]
    lm = modeling_gemma.GemmaForCausalLM(modeling_gemma.GemmaConfig(**c))
    names = [n for n, _ in _lib.GemmaLayer._fields_]
    lm._packed = dict(layers=[{n: torch.zeros(1) for n in names} for _ in range(c["num_hidden_layers"])], inv_freq=torch.zeros(32), norm_w=torch.zeros(1),
                      head_w=torch.zeros(c["vocab_size"], c["hidden_size"], dtype=torch.bfloat16), head_b=torch.zeros(c["vocab_size"]))
    monkeypatch.setattr(_lib, "gemm", lambda *a, **k: None)
    S, W = 5, c["num_key_value_heads"] * c["head_dim"]
    kv = modeling_gemma.KVCache()
    kv._geom = (4, layers, c["num_key_value_heads"], c["head_dim"])
    kv.k_pages, kv.v_pages = torch.zeros(layers, 4, 64, W, dtype=torch.bfloat16), torch.zeros(layers, 4, 64, W, dtype=torch.bfloat16)

    def run():
        return lm.prefill(torch.zeros(S, c["hidden_size"]), torch.arange(S, dtype=torch.int32), 1, S, kv, last_only=True, page_rows=torch.zeros(1, 1, dtype=torch.int32))

    if accepted:
        run()
        assert "pg_gemma_prefill_layers" in library.calls
    else:
        with pytest.raises(ValueError):
            run()
        assert not library.calls


def test_keys_values_and_counters_are_blocks_of_their_own(monkeypatch):
    """Each is as large as it says, so that saving or freeing one does not take or keep another's memory."""
    zeros, arange = torch.zeros, torch.arange
    monkeypatch.setattr(torch, "zeros", lambda *a, device=None, **k: zeros(*a, **k))
    monkeypatch.setattr(torch, "arange", lambda *a, device=None, **k: arange(*a, **k))
    kv = modeling_gemma.KVCache()
    kv.allocate(2, 3, 1, 16, 100)
    for t in (kv.k_pages, kv.v_pages, kv.counters, kv._first_slot):
        assert t.untyped_storage().nbytes() == t.numel() * t.element_size() and not t.any()
    assert kv.k_pages.shape == kv.v_pages.shape == (3, 4, 64, 16) and kv.counters.shape == (3, 2)


def test_a_cache_saved_before_it_had_first_slots_is_read():
    kv = modeling_gemma.KVCache.__new__(modeling_gemma.KVCache)
    kv.__dict__.update(reserve_tokens=4, _geom=None)
    assert kv._first_slot is None
