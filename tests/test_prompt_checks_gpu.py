"""The merge of prompts with their checks inside: flags of every row, rows of ids outside the vocabulary, the first image feature's row; and the errors that a user gets, eager and replayed."""
import copy

import pytest
import torch

from paligemma_multimodal_system_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,N", [(1, 9, 4), (3, 70, 64), (2, 1500, 1024)])
def test_scan_and_text(B, S, N):
    V, D, IMG, PAD = 500, 64, 499, 0
    g = torch.Generator(device="cuda").manual_seed(S)
    ids = torch.randint(1, V - 1, (B, S), generator=g, device="cuda")
    ids[:, 1:1 + N], ids[:, -1] = IMG, PAD
    mask = torch.ones_like(ids)
    mask[:, -1] = 0
    if B > 1:
        ids[1, 1] = 5               # one image token too few
        ids[B - 1, 0] = -3 if B > 2 else V
    embed = torch.randn(V, D, generator=g, device="cuda").to(torch.bfloat16)
    new = [torch.full((B * S,), 77, device="cuda", dtype=torch.int32) for _ in range(2)]
    old = [t.clone() for t in new]
    dst, dst_old = torch.full((B * N,), 77, device="cuda", dtype=torch.int32), torch.full((B * N,), B * S, device="cuda", dtype=torch.int32)
    flags, err = torch.full((B,), 77, device="cuda", dtype=torch.int32), torch.zeros(1, device="cuda", dtype=torch.int32)
    L, st = _lib.lib(), _lib.stream()
    _lib.check(L.pg_prompt_scan(ids.data_ptr(), mask.data_ptr(), new[0].data_ptr(), new[1].data_ptr(), dst.data_ptr(), flags.data_ptr(), B, S, N, V, IMG, PAD, st), "scan")
    _lib.check(L.pg_merge_scan(ids.data_ptr(), mask.data_ptr(), old[0].data_ptr(), old[1].data_ptr(), dst_old.data_ptr(), err.data_ptr(), B, S, N, IMG, PAD, st), "scan")
    assert all(torch.equal(a, b) for a, b in zip(new, old)) and torch.equal(dst, dst_old)
    want = [(int((ids[b] == IMG).sum()) != N) + 2 * int(((ids[b] < 0) | (ids[b] >= V)).any()) for b in range(B)]
    assert flags.tolist() == want and bool(err.item()) == any(w & 1 for w in want)
    h = torch.randn(B * S, D, generator=g, device="cuda")
    before, first = h.clone(), torch.empty(B, 1, D, device="cuda")
    _lib.check(L.pg_prompt_text(ids.data_ptr(), new[1].data_ptr(), dst.data_ptr(), embed.data_ptr(), h.data_ptr(), first.data_ptr(), B, S, D, N, V, 2.0, st), "text")
    flat = ids.view(-1)
    inside = (flat >= 0) & (flat < V)
    text = torch.where((inside & (flat != PAD))[:, None], 2.0 * embed[flat.clamp(0, V - 1)].float(), 0.0)
    assert torch.equal(h, torch.where((flat == IMG)[:, None], before, text))
    assert torch.equal(first[0, 0], before[int(dst[0])])


@pytest.mark.parametrize("replayed", [False, True])
def test_errors(replayed):
    from paligemma_multimodal_system_b200.modeling_paligemma import KVCache, PaliGemmaConfig, PaliGemmaForConditionalGeneration
    from paligemma_multimodal_system_b200.random_init import TINY_CONFIG, make_inputs, make_state_dict
    model = PaliGemmaForConditionalGeneration(PaliGemmaConfig(**copy.deepcopy(TINY_CONFIG)), device="cuda", dtype=torch.bfloat16).eval()
    model.load_state_dict(make_state_dict(TINY_CONFIG, "R1", seed=3), strict=True)
    model.tie_weights()
    inp = {k: v.cuda() for k, v in make_inputs(TINY_CONFIG, batch=2, prompt_len=4, seed=5).items() if torch.is_tensor(v)}
    ids, px, mask = inp["input_ids"], inp["pixel_values"], inp["attention_mask"]

    def call(i):
        if replayed:
            return model.generate(i, px, mask, 2)
        return model(input_ids=i, pixel_values=px, attention_mask=mask, kv_cache=KVCache(), last_only=True)["logits"]

    good = [call(ids).clone() for _ in range(3)]
    for at, value, error in (((1, -2), model.text_config.vocab_size, IndexError), ((0, -1), -1, IndexError), ((1, 0), 5, ValueError)):
        bad = ids.clone()
        bad[at] = value
        with pytest.raises(error):
            call(bad)
    assert torch.equal(call(ids), good[-1])


def _tiny():
    from paligemma_multimodal_system_b200.modeling_paligemma import PaliGemmaConfig, PaliGemmaForConditionalGeneration
    from paligemma_multimodal_system_b200.random_init import TINY_CONFIG, make_inputs, make_state_dict
    model = PaliGemmaForConditionalGeneration(PaliGemmaConfig(**copy.deepcopy(TINY_CONFIG)), device="cuda", dtype=torch.bfloat16).eval()
    model.load_state_dict(make_state_dict(TINY_CONFIG, "R1", seed=3), strict=True)
    model.tie_weights()
    inp = {k: v.cuda() for k, v in make_inputs(TINY_CONFIG, batch=2, prompt_len=4, seed=5).items() if torch.is_tensor(v)}
    return model, inp["input_ids"], inp["pixel_values"], inp["attention_mask"]


@pytest.mark.parametrize("dtype,pitch", [(torch.float32, 1), (torch.float32, 3), (torch.bfloat16, 1), (torch.float64, 2)])
def test_the_first_image_row_goes_to_any_tensor(dtype, pitch):
    model, ids, px, mask = _tiny()
    D = model.text_config.hidden_size
    first = torch.empty(2, 1, D, device="cuda")
    h, _ = model._embed_prompt(ids, mask, px, first_image_row=first)
    room = torch.full((2, pitch, D), 7.0, device="cuda", dtype=dtype)
    model._embed_prompt(ids, mask, px, first_image_row=room[:, :1])
    at = (ids == model.dummy_image_token_id).int().argmax(1)
    assert torch.equal(first[:, 0], h.view(2, -1, D)[torch.arange(2, device="cuda"), at])
    assert torch.equal(room[:, 0], first[:, 0].to(dtype)) and (room[:, 1:] == 7).all()
