"""Prefill attention whose CTAs take several blocks: one round and less, several rounds, last rounds split into single query tiles (with and without a second tile), ragged problems of
different tile counts, both ways of summing rows; against 64-bit sums.  P and V are bf16 (2^-9 each) and the scores' exponentials good to 2^-13: 2^-7 of the values' scale."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,N,dh", [(1, 3, 129, 72), (1, 16, 256, 72), (12, 16, 200, 72), (19, 16, 300, 72), (5, 16, 520, 64), (40, 16, 100, 72), (2, 75, 130, 64)])
@pytest.mark.parametrize("ragged", [False, True])
def test_blocks(B, H, N, dh, ragged):
    from paligemma_multimodal_system_b200 import _lib
    D = H * dh
    g = torch.Generator(device="cuda").manual_seed(N)
    qkv = torch.randn(B * N, 3 * D, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((B * N, D), float("nan"), device="cuda", dtype=torch.bfloat16)
    lens = torch.tensor([1 + (37 * i) % N if ragged else N for i in range(B)], device="cuda", dtype=torch.int32)
    args = (B, H, N, N, dh, 1, N * 3 * D, 3 * D, 0, dh, N * 3 * D, 3 * D, dh, N * D, D, 0, dh, dh ** -0.5, _lib.stream())
    ptrs = (qkv.data_ptr(), qkv.data_ptr() + 2 * D, qkv.data_ptr() + 4 * D, out.data_ptr())
    if ragged:
        _lib.check(_lib.lib().pg_attention_prefill_varlen(*ptrs, lens.data_ptr(), *args), "prefill")
    else:
        _lib.check(_lib.lib().pg_attention_prefill(*ptrs, *args), "prefill")
    for b in range(B):
        n = int(lens[b])
        q, k, v = qkv[b * N:(b + 1) * N].double().view(N, 3, H, dh).permute(1, 2, 0, 3)
        want = torch.softmax(q @ k[:, :n].transpose(1, 2) * dh ** -0.5, -1) @ v[:, :n]
        got = out[b * N:(b + 1) * N].double().view(N, H, dh).transpose(0, 1)
        assert (got[:, :n] - want[:, :n]).abs().max() <= 2.0 ** -7 * max(1.0, want.abs().max().item())


def test_blocks_of_wide_heads():
    from paligemma_multimodal_system_b200 import _lib
    B, S, Hq, dh = 30, 150, 8, 256
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(B * S, n * dh, generator=g, device="cuda").to(torch.bfloat16) for n in (Hq, 1, 1))
    out = torch.full_like(q, float("nan"))
    _lib.check(_lib.lib().pg_attention_prefill(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), B, 1, S * Hq, S, dh, Hq, S * Hq * dh, Hq * dh, dh, 0, S * dh, dh, 0, S * Hq * dh,
                                               Hq * dh, dh, 0, dh ** -0.5, _lib.stream()), "prefill")
    for b in range(B):
        r = slice(b * S, (b + 1) * S)
        want = torch.softmax(q[r].double().view(S, Hq, dh).transpose(0, 1) @ k[r].double().T * dh ** -0.5, -1) @ v[r].double()
        assert (out[r].double().view(S, Hq, dh).transpose(0, 1) - want).abs().max() <= 2.0 ** -7 * max(1.0, want.abs().max().item())
