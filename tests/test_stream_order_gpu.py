"""Calls on one stream with nothing between them, where the later one reads early: products ask for their weight operand and the fused decode attention for its pages
ahead of their dependency wait, the row kernels launch with their descriptors.  Whatever the call in front writes has to be there all the same."""
import math

import pytest
import torch

from paligemma_multimodal_system_b200 import _lib, seq_ops

pytestmark = pytest.mark.gpu


def _t(*shape, seed, dtype=torch.float32, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _queued(calls, rounds=20):
    """The calls back to back, `rounds` times, behind a kernel that keeps the GPU busy until all of them are issued."""
    torch.cuda.synchronize()
    torch.cuda._sleep(4000000)
    for _ in range(rounds):
        for c in calls:
            c()
    torch.cuda.synchronize()


D = 1024


def _producers():
    """name -> (call that writes bf16 rows of the buffer it is given, from inputs that `seed` makes)"""
    w, one = _t(D, seed=1), torch.ones(D, device="cuda")

    def layernorm(out, seed):
        x = _t(out.shape[0], D, seed=seed)
        return lambda: _lib.layernorm(x, w, one, 1e-6, out, None)

    def rmsnorm(out, seed):
        x = _t(out.shape[0], D, seed=seed)
        return lambda: seq_ops.group_rmsnorm_add(x, w, None, out, 1, 1e-6)

    def gate(out, seed):
        x, g = _t(out.shape[0], D, seed=seed), _t(out.shape[0], D, seed=seed + 1, dtype=torch.bfloat16)
        return lambda: seq_ops.rmsnorm_gate(x, w, g, out, 1e-6)

    def embed(out, seed):
        table, tokens = _t(out.shape[0], D, seed=seed, dtype=torch.bfloat16), torch.arange(out.shape[0], device="cuda", dtype=torch.int32)
        return lambda: seq_ops.embed_rows(tokens, table, 0, D, 1.5, out_act=out)

    def geglu(out, seed):
        gu = _t(out.shape[0], 2 * D, seed=seed, dtype=torch.bfloat16)
        return lambda: _lib.check(_lib.lib().pg_geglu(gu.data_ptr(), 2 * D, out.data_ptr(), D, out.shape[0], D, 0, _lib.stream()), "geglu")

    return dict(layernorm=layernorm, rmsnorm=rmsnorm, gate=gate, embed=embed, geglu=geglu)


@pytest.mark.parametrize("name", ["layernorm", "rmsnorm", "gate", "embed", "geglu"])
@pytest.mark.parametrize("T", [5, 300, 2100])
@pytest.mark.parametrize("link", [False, True])
def test_a_product_of_rows_that_the_call_in_front_made(name, T, link):
    """w of the product is the output of the call in front (link: of the one before that); two contents in turn, so that an early read finds the other one."""
    F = 2048
    x, w = _t(T, D, seed=3, dtype=torch.bfloat16, scale=D ** -0.5), torch.empty(F, D, device="cuda", dtype=torch.bfloat16)
    make = _producers()[name]
    a, b = make(w, 10), make(w, 20)
    other, norm_w = _t(64, D, seed=4), torch.ones(D, device="cuda")
    spare = torch.empty(64, D, device="cuda", dtype=torch.bfloat16)
    outs = [torch.empty(T, F, device="cuda") for _ in range(2)]
    calls = []
    for fill, out in zip((a, b), outs):
        calls.append(fill)
        if link:
            calls.append(lambda: seq_ops.group_rmsnorm_add(other, norm_w, None, spare, 1, 1e-6))
        calls.append(lambda out=out: seq_ops.linear(x, w, out))
    _queued(calls)
    for fill, out in zip((a, b), outs):
        fill()
        torch.cuda.synchronize()
        want = torch.empty(T, F, device="cuda")
        seq_ops.linear(x, w, want)
        torch.cuda.synchronize()
        assert (out - want).abs().max().item() <= 1e-4 * want.abs().max().item()  # (split K may add its parts in any order)


def test_the_engine_takes_its_promise_back():
    """Products of a model's step have weights behind them and say so; a step that fails must not leave that said."""
    from paligemma_multimodal_system_b200.engine import SequenceEngine

    class Broken:
        vocab_size, prec = 8, seq_ops.Precision(torch.bfloat16)

        def cache_layout(self):
            from paligemma_multimodal_system_b200.mixers import WindowedSoftmaxAttention
            return [WindowedSoftmaxAttention(64, 2, 1, 32, 32, 1.0, 1e-5).cache_spec()]

        def step(self, *a, **k):
            raise RuntimeError("broken")

    with pytest.raises(RuntimeError, match="broken"):
        SequenceEngine(Broken(), 128, 1).step([("a", [1, 2], [1])])
    for name in ("rmsnorm", "gate", "embed"):
        test_a_product_of_rows_that_the_call_in_front_made(name, 300, False)


def test_norm_weights_that_the_product_in_front_made():
    """w of a norm is the fp32 row of the product in front."""
    x, w = _t(2, 512, seed=5, dtype=torch.bfloat16), _t(D, 512, seed=6, dtype=torch.bfloat16, scale=512 ** -0.5)
    y, row = _t(32, D, seed=7), torch.zeros(1, D, device="cuda")
    acts = [torch.empty(32, D, device="cuda") for _ in range(2)]
    calls = []
    for i in range(2):
        calls.append(lambda i=i: seq_ops.linear(x[i:i + 1], w, row))
        calls.append(lambda i=i: seq_ops.group_rmsnorm_add(y, row.view(-1), None, acts[i], 1, 1e-6))
    _queued(calls)
    yd = y.double()
    for i in range(2):
        want = yd / torch.sqrt((yd * yd).mean(-1, keepdim=True) + 1e-6) * (x[i:i + 1].double() @ w.double().T)
        assert (acts[i].double() - want).abs().max().item() <= 1e-4 * want.abs().max().item()


@pytest.mark.parametrize("B,Hq,dh,L", [(4, 8, 256, 300), (64, 8, 256, 130), (2, 4, 64, 700)])
def test_fused_decode_attention_behind_the_append(B, Hq, dh, L):
    """pg_rope_kv_append writes a sequence's L rows, pg_attention_decode_fused follows with its next token: against the same two calls with a synchronisation between
    them, and against plain softmax on the host."""
    page = 64
    per = L // page + 1
    table = torch.arange(B * per, device="cuda", dtype=torch.int32).view(B, per).flip(1).contiguous()
    kp, vp = (torch.zeros(B * per, page, dh, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    inv = torch.zeros(dh // 2, device="cuda")  # (no rotation: what is checked is the order)
    pos, base = torch.zeros(B * L, device="cuda", dtype=torch.int32), torch.zeros(B, device="cuda", dtype=torch.int32)
    kv_len = torch.full((B,), L + 1, device="cuda", dtype=torch.int32)
    rows = [_t(B * L, 2 * dh, seed=s, scale=0.5) for s in (8, 9)]
    new = _t(B, (Hq + 2) * dh, seed=10, scale=0.5)
    outs = [torch.empty(B, Hq * dh, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    dummy, lib = torch.empty(1, device="cuda", dtype=torch.bfloat16), _lib.lib()

    def append(r):
        _lib.check(lib.pg_rope_kv_append(r.data_ptr(), 1, pos.data_ptr(), dummy.data_ptr(), 0, 0, kp.data_ptr(), vp.data_ptr(), table.data_ptr(), base.data_ptr(), B, L, 0, 1, dh,
                                         page, per, inv.data_ptr(), _lib.stream()), "append")

    def attend(out):
        _lib.check(lib.pg_attention_decode_fused(new.data_ptr(), pos.data_ptr(), kv_len.data_ptr(), inv.data_ptr(), kp.data_ptr(), vp.data_ptr(), table.data_ptr(),
                                                 out.data_ptr(), B, Hq, 1, dh, page, B * per, per, 1.0 / math.sqrt(dh), _lib.stream()), "attention")

    _queued([c for r, o in zip(rows, outs) for c in (lambda r=r: append(r), lambda o=o: attend(o))])
    for r, o in zip(rows, outs):
        append(r)
        torch.cuda.synchronize()
        again = torch.empty_like(o)
        attend(again)
        torch.cuda.synchronize()
        assert torch.equal(o, again)
        kv = torch.cat([r.cpu().bfloat16().float().view(B, L, 2, dh), new.cpu()[:, Hq * dh:].bfloat16().float().view(B, 1, 2, dh)], 1)
        q = new.cpu()[:, :Hq * dh].bfloat16().float().view(B, Hq, dh)
        want = torch.softmax(q @ kv[:, :, 0].transpose(1, 2) / math.sqrt(dh), -1) @ kv[:, :, 1]
        assert (o.cpu().float().view(B, Hq, dh) - want).abs().max() <= 1.5e-2 * want.abs().max()


@pytest.mark.parametrize("B,Hq,dh,L", [(4, 8, 256, 300), (64, 8, 256, 130), (2, 4, 64, 700)])
def test_fused_decode_attention_behind_the_rows_of_a_prompt(B, Hq, dh, L):
    """pg_attn_prepare writes pages, the fused decode attention reads pages ahead of its wait: in order also where the products are promised to take weights."""
    page = 64
    per = L // page + 1
    table = torch.arange(B * per, device="cuda", dtype=torch.int32).view(B, per).flip(1).contiguous()
    kp, vp = (torch.zeros(B * per, page, dh, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    entry, at = torch.arange(B, device="cuda", dtype=torch.int32).repeat_interleave(L), torch.arange(L, device="cuda", dtype=torch.int32).repeat(B)
    freq, inv = torch.zeros(1, device="cuda", dtype=torch.float64), torch.zeros(dh // 2, device="cuda")
    pos, kv_len = torch.zeros(B, device="cuda", dtype=torch.int32), torch.full((B,), L + 1, device="cuda", dtype=torch.int32)
    rows = [_t(B * L, (Hq + 2) * dh, seed=s, scale=0.5, dtype=torch.bfloat16) for s in (8, 9)]
    q = torch.empty(B * L, Hq * dh, device="cuda", dtype=torch.bfloat16)
    new = _t(B, (Hq + 2) * dh, seed=10, scale=0.5)
    outs = [torch.empty(B, Hq * dh, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    lib = _lib.lib()

    def prepare(r):
        _lib.check(lib.pg_attn_prepare(r.data_ptr(), r.stride(0), at.data_ptr(), entry.data_ptr(), table.data_ptr(), per, page, freq.data_ptr(), 0, 0, q.data_ptr(), kp.data_ptr(),
                                       vp.data_ptr(), B * L, Hq, 1, dh, dh, 0, 1e-6, 0, 0, 0, 1.0, 0, 0, 0.0, 0, _lib.stream()), "prepare")

    def attend(out):
        _lib.check(lib.pg_attention_decode_fused(new.data_ptr(), pos.data_ptr(), kv_len.data_ptr(), inv.data_ptr(), kp.data_ptr(), vp.data_ptr(), table.data_ptr(),
                                                 out.data_ptr(), B, Hq, 1, dh, page, B * per, per, 1.0 / math.sqrt(dh), _lib.stream()), "attention")

    _lib.check(lib.pg_weights_follow(1), "follow")
    try:
        _queued([c for r, o in zip(rows, outs) for c in (lambda r=r: prepare(r), lambda o=o: attend(o))])
    finally:
        _lib.check(lib.pg_weights_follow(0), "follow")
    for r, o in zip(rows, outs):
        prepare(r)
        torch.cuda.synchronize()
        again = torch.empty_like(o)
        attend(again)
        torch.cuda.synchronize()
        assert torch.equal(o, again)
    assert not torch.equal(outs[0], outs[1])
