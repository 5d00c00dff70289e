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


def _fma(a, b, c):  # one rounding (24-bit factors: the product is exact in 64 bits)
    return (a.double() * b.double() + c.double()).float()


@pytest.mark.parametrize("H,dh", [(4, 72), (8, 256)])
def test_every_probability_keeps_its_form(H, dh):
    """One-hot keys and values show the probabilities themselves.  Of every eight scores of a 72-wide head the last three take the polynomial, whatever they are paired with; the row sums
    of a 256-wide head are added in the order of the keys, two at a time."""
    from paligemma_multimodal_system_b200 import _lib
    N, S, D = 256, 64, H * dh
    g = torch.Generator(device="cuda").manual_seed(dh)
    q = (torch.randn(N, H, dh, generator=g, device="cuda") * 12).to(torch.bfloat16)
    eye = torch.eye(S, dh, device="cuda", dtype=torch.bfloat16)
    out = torch.empty(N, H, dh, device="cuda", dtype=torch.bfloat16)
    if dh == 72:
        kv = eye.view(S, 1, dh).expand(S, H, dh).contiguous()
        args = (1, H, N, S, dh, 1, N * D, D, 0, dh, S * D, D, dh, N * D, D, 0, dh)
    else:
        kv = eye
        args = (1, 1, N * H, S, dh, H, N * D, D, dh, 0, S * dh, dh, 0, N * D, D, dh, 0)
    scale = dh ** -0.5
    _lib.check(_lib.lib().pg_attention_prefill(q.data_ptr(), kv.data_ptr(), kv.data_ptr(), out.data_ptr(), *args, scale, _lib.stream()), "prefill")
    f32 = lambda v: torch.tensor(v, device="cuda", dtype=torch.float32)
    unit = f32(scale) * f32(1.4426950408889634)
    s = q[..., :S].float()
    x = _fma(s, unit, -(s.amax(-1, keepdim=True) * unit))
    p = torch.exp2(x)
    if dh == 72:
        c = x.clamp(min=-126.0)
        t = c + 12582912.0
        f = c - (t - 12582912.0)
        y = _fma(_fma(_fma(f32(0.05518874), f, f32(0.24261212)), f, f32(0.69325641)), f, f32(0.99992746))
        p = torch.where(torch.arange(S, device="cuda") % 8 >= 5, y * torch.exp2(t - 12582912.0), p)
        total = p.to(torch.bfloat16).double().sum(-1).float()  # (on the tensor cores, which cut sums off: a last bit now and then)
    else:
        total = torch.zeros_like(p[..., 0])
        for j in range(0, S, 2):
            total = total + (p[..., j] + p[..., j + 1])
    want = (p.to(torch.bfloat16).float() * (1.0 / total)[..., None]).to(torch.bfloat16)
    # a score in the other form rounds elsewhere in one of a hundred cases, two sums side by side in one of a thousand rows; a last bit of the sum in one of 2^15
    assert (out[..., :S] != want).float().mean() <= (1e-3 if dh == 72 else 0.0)


@pytest.mark.parametrize("dh,S", [(256, 263), (256, 40), (72, 200)])
def test_a_block_alone_is_as_among_others(dh, S):
    """One round (256-wide heads: a kernel without the loop over blocks) and several give the same bits, with stamps and without."""
    from paligemma_multimodal_system_b200 import _lib
    L, B, H = _lib.lib(), 40, 8
    g = torch.Generator(device="cuda").manual_seed(S)
    kvh = 1 if dh == 256 else H
    q, k, v = (torch.randn(B * S, n * dh, generator=g, device="cuda").to(torch.bfloat16) for n in (H, kvh, kvh))

    def go(batch):
        out = torch.full_like(q[: batch * S], float("nan"))
        if dh == 256:
            args = (batch, 1, S * H, S, dh, H, S * H * dh, H * dh, dh, 0, S * dh, dh, 0, S * H * dh, H * dh, dh, 0)
        else:
            args = (batch, H, S, S, dh, 1, S * H * dh, H * dh, 0, dh, S * H * dh, H * dh, dh, S * H * dh, H * dh, 0, dh)
        _lib.check(L.pg_attention_prefill(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), *args, dh ** -0.5, _lib.stream()), "prefill")
        return out

    one, all_ = go(1), go(B)
    assert one.isfinite().all() and torch.equal(one, all_[:S])
    stamps = torch.zeros(3 * 32 * 8, device="cuda", dtype=torch.int64)
    try:
        L.pg_debug_set_attn_prefill_trace(stamps.data_ptr())
        again = go(1), go(B)
        torch.cuda.synchronize()
    finally:
        L.pg_debug_set_attn_prefill_trace(None)
    assert torch.equal(again[0], one) and torch.equal(again[1], all_) and (stamps != 0).any()
